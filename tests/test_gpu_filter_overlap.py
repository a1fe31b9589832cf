"""Filters whose output buffer overlaps the input: the result of separate buffers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [130, 257])
@pytest.mark.parametrize("window", ["FILTER_RAMLAK", "FILTER_COSRAMP"])
# (output type, where it starts in values of its own type, relative to the input's first byte)
@pytest.mark.parametrize("dtype,shift", [("float32", 0), ("float32", 1), ("float32", -3), ("float32", "row"),
                                         ("float32", "-row"), ("bfloat16", 0), ("float16", 0), ("bfloat16", "row"),
                                         ("float16", "-row"), ("bfloat16", "half")])
def test_overlapping_buffers(W, window, dtype, shift):
    import torch

    from fastcone_b200 import _lib, ops

    n, H = 40, 64   # more rows than one pass over the chip holds
    dt = getattr(torch, dtype)
    win = getattr(_lib, window)
    cos = win == _lib.FILTER_RAMLAK
    size = n * H * W
    s = {"row": W, "-row": -W, "half": size // 2}.get(shift, shift)
    p = torch.randn((n, H, W), device="cuda", generator=torch.Generator("cuda").manual_seed(W))
    z = np.full(n, H / 2.0, np.float32)
    plan = ops.FilterPlan(p.shape, out_dtype=dt, window=win)
    ref = plan(p, zorigin=z, D=300.0, cosine_weight=cos)
    pad = 4 * W
    base = torch.zeros(size + 2 * pad, device="cuda")
    src = base[pad:pad + size].view(n, H, W)
    flat = base.view(dt)
    o = pad * (4 // dt.itemsize) + s
    dst = flat[o:o + size].view(n, H, W)

    def run():
        src.copy_(p)
        plan(src, zorigin=z, D=300.0, cosine_weight=cos, out=dst)

    run()
    assert torch.equal(dst, ref)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    base.zero_()
    graph.replay()
    assert torch.equal(dst, ref)
