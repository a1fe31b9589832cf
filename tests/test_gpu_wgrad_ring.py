"""The tensor-core weight gradient's ring of staged rows and its box widths, exactly.

With small integers every product and every partial sum is an integer below 2^24, so FP32
accumulation in any order gives the exact weight gradient.
"""
import pytest

pytestmark = pytest.mark.gpu

# x extents that are multiples of 8, 4, 2 and 1 (voxels per box row), below, at and above one tile;
# y extents of one row, of whole chunks of 32 rows and just past them; planes enough that a thread
# block walks several chunks of one, three and 33 rows (148 blocks)
SHAPES = [(1, 1, 8), (3, 32, 128), (2, 33, 136), (5, 31, 132), (2, 65, 130), (3, 34, 263), (400, 1, 8),
          (500, 3, 12), (310, 33, 10), (330, 2, 5)]


@pytest.mark.parametrize("shape", SHAPES)
def test_integer_weight_gradient_is_exact(shape):
    import torch

    from fastcone_b200 import nn, ops

    nz, ny, nx = shape
    g = torch.Generator(device="cuda").manual_seed(3)
    x, gy = (torch.randint(-2, 3, (nz, ny, 2, nx, 8), device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    dw = nn.conv3d16_wgrad(x, gy)
    ops.sync_status()

    def channels_last(a):  # (z, y, x, 16) in FP64
        return a.permute(0, 1, 3, 2, 4).reshape(nz, ny, nx, 16).double()

    xp = torch.nn.functional.pad(channels_last(x), (0, 0, 1, 1, 1, 1, 1, 1))
    yc = channels_last(gy).reshape(-1, 16)
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        ref = yc.T @ xp[dz:dz + nz, dy:dy + ny, dx:dx + nx].reshape(-1, 16)
        assert torch.equal(dw[t].double(), ref), t
