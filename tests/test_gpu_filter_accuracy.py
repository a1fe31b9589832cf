"""Rounding errors of the row filters against FP64 on smooth rows, where they show: the ramp leaves
little of a smooth row and all of the noise that rounding adds to it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def shadows(n, H, W, seed):
    """Shadows of an ellipsoid with 2 % noise, as a scanner's projections are."""
    import torch

    r = np.random.default_rng(seed)
    w = torch.linspace(-1, 1, W, device="cuda")[None, None, :]
    h = torch.linspace(-1, 1, H, device="cuda")[None, :, None]
    a = torch.tensor(r.uniform(0.5, 0.9, n), device="cuda", dtype=torch.float32)[:, None, None]
    o = torch.tensor(r.uniform(-0.1, 0.1, n), device="cuda", dtype=torch.float32)[:, None, None]
    p = 3.0 * (1 - ((w - o) / a) ** 2 - 0.3 * h ** 2).clamp_(min=0).sqrt_()
    g = torch.Generator("cuda").manual_seed(seed)
    return p * (1.0 + 0.02 * torch.randn(p.shape, device="cuda", generator=g))


def response(W, window):
    """The filter's frequency response (FP64) and its cyclic length."""
    import torch

    from fastcone_b200 import _lib

    L = 2 * W if window == _lib.FILTER_RAMLAK else W
    k = torch.arange(L // 2 + 1, device="cuda", dtype=torch.float64)
    if L == 2 * W:
        f = np.pi * k / L
        f[0] = np.pi * 0.125 / L
    elif window == _lib.FILTER_COSRAMP:
        f = k / W * torch.cos(0.5 * k / W * np.pi / W)
    else:
        f = torch.where(k + 0.5 * W <= W - 1, k / W * torch.exp(-0.5 * ((k + 0.5) / (0.125 * W)) ** 2), 0.0)
    return f, L


def filtered(p, f, L):
    import torch

    return torch.fft.irfft(torch.fft.rfft(p, n=L, dim=-1) * f, n=L, dim=-1)[..., : p.shape[-1]]


def rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("W,D", [(192, 500.0), (192, 256.0), (384, 1000.0), (768, 1000.0), (1536, 2000.0)])
def test_cosine_weight_adds_no_noise(W, D):
    """The kernel's weighting errs no more than FP64 weights whose products are rounded once do, by
    more than 5 %: emulated on the host the weight's own rounding adds at most 2.5 % to the filtered
    rows' error, a reciprocal square root by a plain Newton step 6 to 11 %."""
    import torch

    from fastcone_b200 import _lib, ops

    n, H = 24, 128
    p = shadows(n, H, W, W)
    z = np.full(n, H / 2.0, np.float32)
    ww = torch.arange(W, device="cuda", dtype=torch.float64) - W / 2.0
    hh = (torch.arange(H, device="cuda", dtype=torch.float64) - H / 2.0)[:, None]
    w64 = p.double() * (D / torch.sqrt(D * D + hh * hh + ww * ww))
    want = filtered(w64, *response(W, _lib.FILTER_RAMLAK))
    plan = ops.FilterPlan(p.shape)
    once = rel(plan(w64.float(), cosine_weight=False), want)
    got = rel(plan(p, zorigin=z, D=D), want)
    assert got <= 1.05 * once, (got, once)


@pytest.mark.parametrize("W", [53, 97, 113, 129, 192, 369, 949, 1000, 1411, 4096])
@pytest.mark.parametrize("window", ["FILTER_COSRAMP", "FILTER_GAUSSRAMP"])
def test_unpadded_windows_as_near_as_the_cyclic_transform(W, window):
    """Cyclic filters err no more than FP32 transforms of the rows themselves do; 20 % covers another
    choice of transform for another number of rows."""
    from fastcone_b200 import _lib, ops

    win = getattr(_lib, window)
    p = shadows(16, 128, W, W)
    f, L = response(W, win)
    want = filtered(p.double(), f, L)
    plain = rel(filtered(p, f.float(), L), want)
    got = rel(ops.FilterPlan(p.shape, window=win)(p, cosine_weight=False), want)
    assert got <= 1.2 * plain, (got, plain)
