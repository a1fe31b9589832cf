"""The staged adjoint's padded brick planes: both flushes against the direct scatter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# pixel pitches that give brick rows of different pitches (hence paddings of 0 to 12 words)
CASES = [(0.6, 64), (0.9, 64), (1.0, 64), (1.15, 48), (1.3, 32)]


@pytest.mark.parametrize("flush4", ["1", "0"])
@pytest.mark.parametrize("pw,n", CASES)
def test_adjoint_matches_the_direct_scatter(pw, n, flush4, monkeypatch):
    import torch

    from fastcone_b200 import ConeGeometry, _lib, ops

    views = 12
    ang = (np.arange(views) * (2 * np.pi / views)).astype(np.float32)
    g = ConeGeometry((n, n, 40), (int(1.5 * n / pw), int(44 / pw)), ang, 4.0 * n, pw)
    gen = torch.Generator(device="cuda").manual_seed(2)
    y = torch.rand(g.proj_shape, device="cuda", generator=gen)
    monkeypatch.setenv("FCB_PROJ_FLUSH4", flush4)
    a = ops.ProjectPlan(g).adjoint(y)
    monkeypatch.setenv("FCB_PROJ_NOBRICK", "1")
    b = ops.ProjectPlan(g, method=_lib.PROJ_EXPLICIT_GLOBAL).adjoint(y)
    ops.sync_status()
    # every addend is >= 0 and rounded alike; only the order of a voxel's sum differs: at most
    # N roundings of half an ulp on either side, N = rays within a voxel's support (a square of
    # 2 sqrt(2) voxels, pixels of >= 0.75 pw there) x 4 samples x views
    N = views * 4 * (2 * 2 ** 0.5 / (0.75 * pw) + 1) ** 2
    assert ((a - b).abs() <= 2 * N * 2.0 ** -24 * b + 1e-30).all()
    assert float(b.min()) >= 0 and float(b.max()) > 0
