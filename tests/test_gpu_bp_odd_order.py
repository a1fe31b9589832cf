"""Odd-row plans made and run on side streams: the launches carry their view matrices, so nothing
has to be ordered with another stream, and nothing waits for the device."""
import numpy as np
import pytest

from tests._cases import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_made_and_run_beside_busy_copies(dtype):
    import torch

    from fastcone_b200 import ops

    # 650 views: four launches
    g, _ = make_case(vol_xyz=(40, 33, 35), det_wh=(71, 48), nviews=650, D=160.0, pw=0.8)
    dt = getattr(torch, dtype)
    proj = torch.randn(g.proj_shape, device="cuda").to(dt)
    ref = ops.BackprojectPlan(g, mode=2, dtype=dt)(proj, torch.zeros(g.vol_shape, device="cuda"))
    host = torch.empty(64 << 20, dtype=torch.float32, pin_memory=True)
    dev = torch.empty(64 << 20, dtype=torch.float32, device="cuda")
    copies, s = torch.cuda.Stream(), torch.cuda.Stream()
    a, b = torch.empty_like(ref), torch.empty_like(ref)
    torch.cuda.synchronize()
    for _ in range(4):
        with torch.cuda.stream(copies):
            for _ in range(4):
                dev.copy_(host, non_blocking=True)
        with torch.cuda.stream(s):
            a.zero_()
            b.zero_()
            plan = ops.BackprojectPlan(g, mode=2, dtype=dt)
            plan(proj, a)
            del plan
            ops.backproject(proj, g, vol=b)
        torch.cuda.synchronize()
        assert torch.equal(a, ref) and torch.equal(b, ref)


def test_one_shot_call_does_not_wait_for_other_streams():
    import torch

    from fastcone_b200 import ops

    g, _ = make_case(vol_xyz=(40, 33, 35), det_wh=(71, 48), nviews=60, D=160.0, pw=0.8)
    proj = torch.randn(g.proj_shape, device="cuda")
    vol = torch.zeros(g.vol_shape, device="cuda")
    busy, s = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(s):
        ops.backproject(proj, g, vol=vol)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(2_000_000_000)  # about a second
        done.record()
    with torch.cuda.stream(s):
        ops.backproject(proj, g, vol=vol)
    returned_first = not done.query()
    torch.cuda.synchronize()
    assert returned_first


@pytest.mark.parametrize("views", [300, 301, 900])
def test_launches_of_many_views(views, monkeypatch):
    """More views per launch than its parameters hold in both forms go in pieces."""
    import torch

    from fastcone_b200 import ops

    monkeypatch.setenv("FCB_FDK_SPLIT", "1")
    g, _ = make_case(vol_xyz=(20, 18, 17), det_wh=(41, 24), nviews=views, D=90.0, pw=0.8)
    proj = torch.randn(g.proj_shape, device="cuda")
    ref = ops.BackprojectPlan(g, mode=2)(proj, torch.zeros(g.vol_shape, device="cuda"))
    monkeypatch.setenv("FCB_FDK_VIEWS", "900")
    got = ops.BackprojectPlan(g, mode=2)(proj, torch.zeros(g.vol_shape, device="cuda"))
    ops.sync_status()
    # the same terms in other partial sums: a rounding per term at most, random signs
    assert float((got - ref).abs().max()) < 64 * 2.0 ** -24 * 4.0 * np.sqrt(views)


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("vol,views", [((33, 30, 27), 250), ((64, 64, 64), 181)])
def test_captured_calls_agree_to_rounding(vol, views, dtype):
    """A captured call runs the generic kernel, which adds the views in one order; an eager call of few
    tiles adds them in the parts of a cluster's CTAs: equal but for the rounding of the sums."""
    import torch

    from fastcone_b200 import ops

    g, _ = make_case(vol_xyz=vol, det_wh=(97, 50), nviews=views, D=260.0, pw=0.8)
    dt = getattr(torch, dtype)
    proj = torch.randn(g.proj_shape, device="cuda").to(dt)
    plan = ops.BackprojectPlan(g, mode=2, dtype=dt)
    eager = plan(proj, torch.zeros(g.vol_shape, device="cuda"))
    out = torch.zeros(g.vol_shape, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan(proj, out)
    out.zero_()
    graph.replay()
    ops.sync_status()
    assert float((eager - out).abs().max()) < 64 * 2.0 ** -24 * 4.0 * np.sqrt(views)
