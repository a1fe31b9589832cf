"""The default convolution kernel's walks (rows and planes per thread block), exactly.

With small integers every partial sum is an integer far below 2^24: FP32 accumulation is exact.
"""
import pytest

pytestmark = pytest.mark.gpu

# one plane, two, and walks whose last plane falls into each of the three accumulator blocks; one row
# to more rows than a walk has; one partial tile, a whole one and two; several walks per block
SHAPES = [(1, 1, 1), (2, 1, 8), (3, 2, 5), (4, 3, 129), (5, 4, 128), (7, 6, 130), (65, 5, 12), (66, 11, 3),
          (67, 7, 33), (90, 131, 131), (130, 200, 6)]


@pytest.mark.parametrize("shape", SHAPES)
def test_integer_convolution_is_exact(shape, monkeypatch):
    import torch

    from fastcone_b200 import nn, ops

    monkeypatch.delenv("FCB_CONV_SIMPLE", raising=False)
    nz, ny, nx = shape
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randint(-2, 3, (nz, ny, 2, nx, 8), device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randint(-2, 3, (27, 16, 16), device="cuda", generator=g).to(torch.bfloat16)
    y = nn.conv3d16(x, w, None, relu=False, out_dtype=torch.float32)
    ops.sync_status()

    def channels_last(a):  # (z, y, x, 16) in FP64
        return a.permute(0, 1, 3, 2, 4).reshape(nz, ny, nx, 16).double()

    xp = torch.nn.functional.pad(channels_last(x), (0, 0, 1, 1, 1, 1, 1, 1))
    ref = torch.zeros((nz, ny, nx, 16), device="cuda", dtype=torch.float64)
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        ref += xp[dz:dz + nz, dy:dy + ny, dx:dx + nx] @ w[t].double().T
    assert torch.equal(channels_last(y), ref)
