"""The batched Katsevich filter: batches of views, aliased buffers and the sizes that leave the
staged and fused forms, against the FP64 restatement (rel-L2 <= 1e-5, the filter's bound)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _geom(W, H, views):
    from fastcone_b200.geometry import ConeGeometry

    return ConeGeometry.helical((48, 48, 40), 1.0, (W, H), 1.0, 150.0, 300.0, 3, views // 3, 24.0)


# odd and unaligned widths; 800 rows: no room to stage a strip; 4100 columns: longer than the row transform
@pytest.mark.parametrize("W,H,views", [(96, 24, 240), (41, 24, 60), (94, 7, 60), (33, 2, 9), (40, 800, 9), (4100, 6, 6)])
@pytest.mark.parametrize("mb", [None, "1"])
def test_filter_sizes_and_batches(W, H, views, mb, monkeypatch):
    import torch

    from fastcone_b200 import ops

    if mb:
        monkeypatch.setenv("FCB_KATS_BATCH_MB", mb)
    g = _geom(W, H, views)
    p = np.random.default_rng(W + H).random(g.proj_shape, dtype=np.float32)
    want = O.katsevich_filter(p, g.angles, g.D, g.pw, g.helical_pitch)
    got = ops.KatsevichPlan(g)(torch.from_numpy(p).cuda()).cpu().numpy()
    assert O.rel_l2(got, want) < 1e-5, O.rel_l2(got, want)


@pytest.mark.parametrize("shift", [0, 1, -1, 5, 1000, -1000])
def test_aliased_buffers(shift, monkeypatch):
    """out == in, and buffers that overlap in another way, give the result of separate ones."""
    import torch

    from fastcone_b200 import ops

    monkeypatch.setenv("FCB_KATS_BATCH_MB", "1")
    g = _geom(96, 24, 240)
    p = torch.rand(g.proj_shape, device="cuda")
    plan = ops.KatsevichPlan(g)
    ref = plan(p.clone())
    n = p.numel()
    buf = torch.zeros(n + 2000, device="cuda")
    a = buf[1000:1000 + n].view(g.proj_shape).copy_(p)
    b = buf[1000 + shift:1000 + shift + n].view(g.proj_shape)
    assert torch.equal(plan(a, out=b), ref) or float((b - ref).norm() / ref.norm()) < 1e-6
