"""Clusters as the default rule chooses them: captured and direct calls, PI window included."""
import pytest

from tests._cases import make_case

pytestmark = pytest.mark.gpu


def _captured(plan, proj, shape):
    import torch

    out = torch.zeros(shape, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan(proj, out)
    out.zero_()
    graph.replay()
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("vol,views", [((33, 30, 27), 250), ((16, 16, 1), 24), ((96, 80, 90), 61), ((160, 160, 150), 40)])
def test_captured_call_repeats_the_direct_one(vol, views, dtype):
    import torch

    from fastcone_b200 import ops

    g, _ = make_case(vol_xyz=vol, det_wh=(vol[0] * 2 // 8 * 8, vol[2] * 3 // 2), nviews=views, D=4.0 * vol[0] + 20, pw=0.8)
    dt = getattr(torch, dtype)
    proj = torch.randn(g.proj_shape, device="cuda").to(dt)
    plan = ops.BackprojectPlan(g, mode=2, dtype=dt)
    ref = plan(proj, torch.zeros(g.vol_shape, device="cuda"))
    assert torch.equal(_captured(plan, proj, g.vol_shape), ref)
    ops.sync_status()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_pi_window(dtype, monkeypatch):
    """Views of half a turn reach a tile: the ranks take every n-th of them."""
    import torch

    from fastcone_b200 import _lib, ops
    from fastcone_b200.geometry import ConeGeometry

    g = ConeGeometry.helical((40, 40, 36), 1.0, (112, 28), 1.0, 150.0, 300.0, 5, 47, 24.0, pi_window=True)
    dt = getattr(torch, dtype)
    proj = torch.randn(g.proj_shape, device="cuda", generator=torch.Generator("cuda").manual_seed(3)).to(dt)
    plan = ops.BackprojectPlan(g, mode=_lib.MODE_KATSEVICH, dtype=dt)
    got = plan(proj, torch.zeros(g.vol_shape, device="cuda"))
    assert torch.equal(_captured(plan, proj, g.vol_shape), got)
    monkeypatch.setenv("FCB_FDK_SPLIT", "1")
    one = plan(proj, torch.zeros(g.vol_shape, device="cuda"))
    ops.sync_status()
    # the same terms, of about 47 / 2 views a voxel, in other partial sums
    assert float((got - one).abs().max()) < 64 * 2.0 ** -24 * 4.0 * 24.0 ** 0.5
