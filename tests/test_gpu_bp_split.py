"""Backprojection with a tile's views shared by a cluster's CTAs, against one CTA per tile: the
same sums in another order."""
import numpy as np
import pytest

from tests._cases import make_case

pytestmark = pytest.mark.gpu

# Sums of n terms split into parts: each part and the sum of the parts round once more per term at
# most, 2^-24 sqrt(n) of the terms' norm for random signs; 64 x that for the largest of the voxels.
TOL = 64 * 2.0 ** -24


def _run(plan, proj, shape, ranks, monkeypatch):
    import torch

    from fastcone_b200 import ops

    monkeypatch.setenv("FCB_FDK_SPLIT", str(ranks))
    # (added to what is there: every plane of the tile is written once)
    out = plan(proj, torch.full(shape, 0.25, device="cuda"))
    ops.sync_status()
    return out - 0.25


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("W", [72, 71])  # aligned rows, repacked rows
@pytest.mark.parametrize("vol,views", [((33, 30, 27), 250), ((16, 16, 1), 8), ((50, 20, 70), 61)])
def test_split_views(vol, views, W, dtype, monkeypatch):
    import torch

    from fastcone_b200 import ops

    g, _ = make_case(vol_xyz=vol, det_wh=(W, 48), nviews=views, D=130.0, pw=0.8)
    dt = getattr(torch, dtype)
    proj = torch.randn(g.proj_shape, device="cuda", generator=torch.Generator("cuda").manual_seed(views)).to(dt)
    plan = ops.BackprojectPlan(g, mode=2, dtype=dt)
    ref = _run(plan, proj, g.vol_shape, 1, monkeypatch)
    scale = float(views) ** 0.5 * 4.0
    for ranks in (2, 3, 5, 6, 7, 8):
        got = _run(plan, proj, g.vol_shape, ranks, monkeypatch)
        assert float((got - ref).abs().max()) < TOL * scale, ranks
        assert torch.equal(got, _run(plan, proj, g.vol_shape, ranks, monkeypatch))  # no dependence on timing


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_split_views_pi_window(dtype, monkeypatch):
    import torch

    from fastcone_b200 import _lib, ops
    from fastcone_b200.geometry import ConeGeometry

    g = ConeGeometry.helical((40, 40, 36), 1.0, (112, 28), 1.0, 150.0, 300.0, 5, 120, 24.0, pi_window=True)
    dt = getattr(torch, dtype)
    proj = torch.randn(g.proj_shape, device="cuda", generator=torch.Generator("cuda").manual_seed(3)).to(dt)
    plan = ops.BackprojectPlan(g, mode=_lib.MODE_KATSEVICH, dtype=dt)
    ref = _run(plan, proj, g.vol_shape, 1, monkeypatch)
    for ranks in (2, 6, 8):
        got = _run(plan, proj, g.vol_shape, ranks, monkeypatch)
        assert float((got - ref).abs().max()) < TOL * 4.0 * 60.0 ** 0.5, ranks


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_split_wait_runs_out(dtype, monkeypatch):
    """A rank whose producer stops early reports the timeout and the cluster still ends."""
    import ctypes

    import torch

    from fastcone_b200 import _lib, ops

    monkeypatch.setenv("FCB_FDK_SPLIT", "6")
    g, _ = make_case(vol_xyz=(33, 30, 27), det_wh=(72, 48), nviews=60, D=130.0, pw=0.8)
    dt = getattr(torch, dtype)
    plan = ops.BackprojectPlan(g, mode=2, dtype=dt)
    _lib.check(_lib.lib().fcb_bp_plan_set_test_stall(plan._h, 3, ctypes.c_ulonglong(20000000)))
    plan(torch.zeros(g.proj_shape, device="cuda", dtype=dt), torch.zeros(g.vol_shape, device="cuda"))
    with pytest.raises(_lib.FastconeError):
        ops.sync_status()
    plan2 = ops.BackprojectPlan(g, mode=2, dtype=dt)
    plan2(torch.zeros(g.proj_shape, device="cuda", dtype=dt), torch.zeros(g.vol_shape, device="cuda"))
    ops.sync_status()
