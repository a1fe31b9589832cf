"""The one-pass incoming gradient of a convolution layer against the element-wise operations it
stands for: the same BF16 values, and sums within FP32 rounding."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 5, 7), (6, 33, 130), (40, 41, 101)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("relu", [False, True])
def test_grad_prep(shape, dtype, relu):
    import torch

    from fastcone_b200 import nn

    nz, ny, nx = shape
    g = torch.Generator(device="cuda").manual_seed(nx)
    gy = torch.randn((nz, ny, 2, nx, 8), device="cuda", generator=g).to(getattr(torch, dtype))
    y = torch.randn(gy.shape, device="cuda", generator=g).relu_().to(torch.bfloat16)
    if nx > 1:  # what is not finite goes through the same products
        gy[0, 0, 0, 0, 0] = float("inf")
        gy[0, 0, 0, 1, 1] = float("nan")
        y[0, 0, 0, 0, 0] = 0.0
        y[0, 0, 1, 0, 0] = float("nan")
    ref = gy.float()
    if relu:
        ref = ref * (y > 0)
    gb, db = nn.conv3d16_grad_prep(gy, y if relu else None)
    assert torch.equal(gb.view(torch.int16), ref.to(torch.bfloat16).view(torch.int16)) or \
        torch.equal(torch.nan_to_num(gb.float(), 7.0), torch.nan_to_num(ref.to(torch.bfloat16).float(), 7.0))
    want = ref.double().sum(dim=(0, 1, 3)).reshape(16)
    # n terms in parts: 2^-24 times the terms' absolute sum bounds each channel's rounding
    bound = ref.double().abs().sum(dim=(0, 1, 3)).reshape(16) * 2.0 ** -24 * 16
    fin = torch.isfinite(want)
    assert torch.equal(fin, torch.isfinite(db))
    assert ((db.double() - want).abs()[fin] <= bound[fin] + 1e-30).all()
    gb2, db2 = nn.conv3d16_grad_prep(gy, y if relu else None)
    assert torch.equal(db.nan_to_num(), db2.nan_to_num())


def test_conv_backward_paths_agree():
    """The one-pass backward and the element-wise one (taken under create_graph) give the same
    gradients."""
    import torch

    from fastcone_b200 import nn

    torch.manual_seed(0)
    layer = nn.Conv3d(16, 16, relu=True).cuda()
    x = torch.randn((9, 10, 2, 70, 8), device="cuda").relu_().to(torch.bfloat16).requires_grad_()
    gy = torch.randn(x.shape, device="cuda").to(torch.bfloat16)
    args = [x, layer.weight, layer.bias]
    a = torch.autograd.grad(layer(x), args, gy)
    b = torch.autograd.grad(layer(x), args, gy, create_graph=True)
    assert torch.equal(a[0], b[0])
    for u, v in zip(a[1:], b[1:]):
        assert float((u - v).norm() / v.norm()) < 2e-6
