"""The Katsevich filter on both sides of the sizes where its derivative gets a pass of its own, against
the FP64 restatement (rel-L2 <= 1e-5, the filter's bound)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,views", [(40, 768, 7), (40, 769, 7), (259, 801, 5), (33, 1025, 4), (4100, 15, 6),
                                       (4100, 16, 6), (4099, 17, 5), (70, 20, 900)])
@pytest.mark.parametrize("mb", [None, "1"])
def test_staged_and_two_pass_sizes(W, H, views, mb, monkeypatch):
    import torch

    from fastcone_b200 import ops
    from fastcone_b200.geometry import ConeGeometry

    if mb:
        monkeypatch.setenv("FCB_KATS_BATCH_MB", mb)
    g = ConeGeometry.helical((48, 48, 40), 1.0, (W, H), 1.0, 150.0, 300.0, 1, views, 24.0)
    p = np.random.default_rng(W + H).random(g.proj_shape, dtype=np.float32)
    want = O.katsevich_filter(p, g.angles, g.D, g.pw, g.helical_pitch)
    plan = ops.KatsevichPlan(g)
    x = torch.from_numpy(p).cuda()
    got = plan(x)
    assert O.rel_l2(got.cpu().numpy(), want) < 1e-5
    assert torch.equal(plan(x, out=x), got)
