"""The Hilbert transform of the Katsevich filter in the row transform's longer shapes, against the FP64
restatement (rel-L2 <= 1e-5, the filter's bound)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [769, 1024, 1025, 1536, 2047, 2049, 3073, 4096])
def test_hilbert_in_long_rows(W):
    import torch

    from fastcone_b200 import ops
    from fastcone_b200.geometry import ConeGeometry

    g = ConeGeometry.helical((48, 48, 40), 1.0, (W, 6), 1.0, 150.0 + W, 300.0 + 2 * W, 1, 9, 24.0)
    p = np.random.default_rng(W).random(g.proj_shape, dtype=np.float32)
    want = O.katsevich_filter(p, g.angles, g.D, g.pw, g.helical_pitch)
    got = ops.KatsevichPlan(g)(torch.from_numpy(p).cuda()).cpu().numpy()
    assert O.rel_l2(got, want) < 1e-5, O.rel_l2(got, want)
