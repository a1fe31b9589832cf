"""The fused row filter at the edges of its transform sizes, against the FP64 restatement."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# Unit roundoff times the radix-2 depth of both transforms of the longest size (2 x 13), with
# a factor of one for the twiddles: 6e-8 x 26 = 1.6e-6 of the result's norm for white input.
TOL = 1.6e-6
# smallest widths, both sides of every transform size, the last fused width and the first long one
WIDTHS = [1, 2, 3, 31, 32, 33, 48, 49, 64, 65, 96, 97, 128, 129, 192, 193, 256, 257, 384, 385, 512, 513, 768, 769,
          1024, 1025, 1536, 1537, 2048, 2049, 3072, 3073, 4096, 4097]


@pytest.mark.parametrize("W", WIDTHS)
def test_row_filter_sizes(W):
    import torch

    from fastcone_b200 import _lib, ops

    # 17 rows per view: the last group of rows of a warp is partly filled at every size
    proj = np.random.default_rng(W).standard_normal((3, 17, W)).astype(np.float32)
    x = torch.from_numpy(proj).cuda()
    for win, want in ((_lib.FILTER_RAMLAK, O.rampfilter(proj.astype(np.float64))),
                      (_lib.FILTER_COSRAMP, O.apodised_rampfilter(proj.astype(np.float64), "cosramp", 0.125))):
        got = ops.FilterPlan(proj.shape, window=win)(x, cosine_weight=False).cpu().numpy()
        if np.abs(want).max() < 1e-12 * np.abs(proj).max():  # a width of 1: nothing but the DC bin
            assert np.abs(got).max() <= 1e-6 * np.abs(proj).max()
        else:
            assert O.rel_l2(got, want) < TOL, (win, O.rel_l2(got, want))


@pytest.mark.parametrize("W", [40, 101, 300, 600, 1536, 2500])
def test_row_filter_rows_are_independent(W):
    """A NaN, an infinity or a huge row changes its own row only, and a zero row stays zero."""
    import torch

    from fastcone_b200 import ops

    p = torch.randn((2, 21, W), device="cuda", generator=torch.Generator("cuda").manual_seed(W))
    plan = ops.FilterPlan(p.shape)
    z = np.full(2, 10.0, np.float32)
    ref = plan(p, zorigin=z, D=300.0)
    q = p.clone()
    q[0, 3, W // 2] = float("nan")
    q[0, 6, W // 3] = float("inf")
    q[1, 7] *= 1e30
    q[1, 12] = 0.0
    got = plan(q, zorigin=z, D=300.0)
    assert not torch.isfinite(got[0, 3]).any() and not torch.isfinite(got[0, 6]).any()
    assert (got[1, 12] == 0).all()
    same = torch.ones((2, 21), dtype=torch.bool)
    same[0, 3] = same[0, 6] = same[1, 7] = same[1, 12] = False
    assert torch.equal(got[same.cuda()], ref[same.cuda()])


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
def test_row_filter_unaligned_buffers(dtype):
    """Buffers that are not aligned to a pair of values give the aligned buffers' result."""
    import torch

    from fastcone_b200 import ops

    dt = getattr(torch, dtype)
    n, H, W = 2, 9, 130
    p = torch.randn((n, H, W), device="cuda")
    plan = ops.FilterPlan((n, H, W), out_dtype=dt)
    z = np.full(n, 4.0, np.float32)
    ref = plan(p, zorigin=z, D=200.0)
    src = torch.empty(n * H * W + 1, device="cuda")[1:].view(n, H, W).copy_(p)
    dst = torch.empty(n * H * W + 1, device="cuda", dtype=dt)[1:].view(n, H, W)
    assert torch.equal(plan(src, zorigin=z, D=200.0, out=dst), ref)
