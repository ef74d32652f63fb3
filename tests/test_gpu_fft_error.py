"""Rounding of the shared-memory transforms on noise, where no large term hides
it: the errors against float64 of the same transform with each stage twiddle
rounded once and each constant of a butterfly in one float (measured, by length,
to 1 %).  Twiddles formed as products of others are a quarter above them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _noise(seed, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda")


def _off(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("N,bound", [(256, 1.80e-7), (512, 1.90e-7), (1024, 1.96e-7), (2048, 2.13e-7)])
def test_sprite_transform(N, bound):
    from ghostlight_gb300.starburst import SpritePlan
    a = _noise(N, N, N)
    plan = SpritePlan(N, np.array([[550.0, 1.0, 1.0, 1.0]], np.float32))
    plan.bake(a, 2)
    psf, _, _ = plan.read()
    want = torch.fft.fftshift(torch.fft.fft2(a.double()).abs() ** 2)
    assert _off(psf, want) < bound
    mc = N // 4
    lags = torch.empty((2 * mc + 1, 2 * mc + 1), device="cuda")
    plan.autocorr(a, mc, lags)
    c = torch.roll(torch.fft.ifft2(torch.fft.fft2(a.double()).abs() ** 2).real, (mc, mc), (0, 1))[:2 * mc + 1, :2 * mc + 1]
    # the zero lag's place holds the scale: float32 sums of N^2 like terms in ~5 levels
    assert float(lags[mc, mc]) * N * N == pytest.approx(1.0, abs=2e-7)
    assert _off(lags * (N * N), c / c[mc, mc]) < 4e-7
    plan.close()
