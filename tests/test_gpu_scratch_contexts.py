"""The scratch pools of two contexts that live side by side on one device."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_alternating_contexts_keep_their_pools():
    """Calls that alternate between the primary context and another one reuse each context's idle
    scratch: the device's free memory settles after the first call in each."""
    import torch

    from fastcone_b200 import _lib, ops
    from fastcone_b200.geometry import ConeGeometry

    cu = ctypes.CDLL("libcuda.so.1")
    n = 192   # 28 MB of scratch a call
    ang = (np.arange(4) * (2 * np.pi / 4)).astype(np.float32)
    g = ConeGeometry((n, n, n), (3 * n // 2, n), ang, 4.0 * n, 1.0)
    vol = torch.rand(g.vol_shape, device="cuda")
    ref = ops.project(vol, g, method=_lib.PROJ_EXPLICIT)
    torch.cuda.synchronize()

    def ok(rc):
        assert rc == 0, rc

    ctx = ctypes.c_void_p()
    ok(cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, torch.cuda.current_device()))
    try:
        # (the new context is current) its own buffers, the same volume
        dv, dp = ctypes.c_uint64(), ctypes.c_uint64()
        ok(cu.cuMemAlloc_v2(ctypes.byref(dv), ctypes.c_size_t(vol.numel() * 4)))
        ok(cu.cuMemAlloc_v2(ctypes.byref(dp), ctypes.c_size_t(ref.numel() * 4)))
        ok(cu.cuMemsetD32_v2(dv, 0, ctypes.c_size_t(vol.numel())))
        ok(cu.cuMemsetD32_v2(dp, 0, ctypes.c_size_t(ref.numel())))
        ok(cu.cuCtxPopCurrent_v2(ctypes.byref(ctypes.c_void_p())))

        gs = g.struct()

        def other():
            ok(cu.cuCtxPushCurrent_v2(ctx))
            try:
                _lib.check(_lib.lib().fcb_project_device(ctypes.byref(gs), _lib.PROJ_EXPLICIT,
                                                         ctypes.c_void_p(dv.value), ctypes.c_void_p(dp.value), None))
                ok(cu.cuCtxSynchronize())
            finally:
                ok(cu.cuCtxPopCurrent_v2(ctypes.byref(ctypes.c_void_p())))

        def free():
            torch.cuda.synchronize()
            return torch.cuda.mem_get_info()[0]

        out = torch.empty_like(ref)

        def primary():
            ops.project(vol, g, method=_lib.PROJ_EXPLICIT, proj=out.zero_())
            torch.cuda.synchronize()

        other()
        primary()
        before = free()
        for _ in range(6):
            other()
            primary()
        assert torch.equal(out, ref)
        assert before - free() < 20 << 20
    finally:
        ok(cu.cuCtxDestroy_v2(ctx))
    # the primary context's pool still serves calls
    assert torch.equal(ops.project(vol, g, method=_lib.PROJ_EXPLICIT), ref)
