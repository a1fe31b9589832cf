"""Backprojection of projections whose rows are not whole 16-byte groups: the staged kernels on
repacked rows give the generic kernel's result (which a captured call still runs), and the FP64
oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from tests._cases import make_case, smooth_projections

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("vol,det,views", [((33, 30, 27), (71, 48), 250), ((17, 40, 65), (53, 31), 21),
                                           ((64, 64, 32), (97, 50), 181), ((16, 16, 1), (33, 9), 1)])
def test_repacked_rows_equal_generic(vol, det, views, mode, dtype, monkeypatch):
    import torch

    # one CTA per tile: the generic kernel's order of additions over the views
    monkeypatch.setenv("FCB_FDK_SPLIT", "1")

    from fastcone_b200 import ops

    g, pb = make_case(vol_xyz=vol, det_wh=det, nviews=views, D=130.0, pw=0.8)
    dt = getattr(torch, dtype)
    proj = torch.randn(g.proj_shape, device="cuda", generator=torch.Generator("cuda").manual_seed(views)).to(dt)
    plan = ops.BackprojectPlan(g, mode=mode, dtype=dt)
    got = plan(proj, torch.zeros(g.vol_shape, device="cuda"))
    ref = torch.zeros(g.vol_shape, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan(proj, ref)
    ref.zero_()
    graph.replay()
    ops.sync_status()
    # the same positions, weights and order of additions; the generic kernel leaves out the views
    # whose taps all lie outside, which add zeros here
    assert torch.equal(got, ref), float((got - ref).abs().max())


@pytest.mark.parametrize("dtype,tol", [("float32", 2e-5), ("bfloat16", 1e-2)])
def test_repacked_rows_vs_oracle(dtype, tol):
    import torch

    from fastcone_b200 import ops

    g, pb = make_case(vol_xyz=(33, 30, 27), det_wh=(71, 48), nviews=190, D=130.0, pw=0.8)
    proj, p64 = smooth_projections(pb)
    dt = getattr(torch, dtype)
    got = ops.backproject(torch.from_numpy(proj).cuda().to(dt), g, mode=2)
    want = O.backproject_f64(pb, proj, kernel_mode=2)
    assert O.rel_l2(got.cpu().numpy(), want) < tol


def test_repacked_rows_on_streams():
    """One plan on several streams at once: each call has its own repacked rows."""
    import torch

    from fastcone_b200 import ops

    g, _ = make_case(vol_xyz=(64, 64, 64), det_wh=(97, 63), nviews=200, D=260.0, pw=0.8)
    plan = ops.BackprojectPlan(g, mode=2)
    projs = [torch.randn(g.proj_shape, device="cuda") for _ in range(4)]
    refs = [plan(p, torch.zeros(g.vol_shape, device="cuda")) for p in projs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in projs]
    outs = [torch.zeros(g.vol_shape, device="cuda") for _ in projs]
    torch.cuda.synchronize()
    for s, p, o in zip(streams, projs, outs):
        with torch.cuda.stream(s):
            plan(p, o)
    torch.cuda.synchronize()
    for o, r in zip(outs, refs):
        assert torch.equal(o, r)
