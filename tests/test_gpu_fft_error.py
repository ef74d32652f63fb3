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


# the error of the same convolution with a kernel spectrum and whole-circle
# twiddles in float32, its best plane (the smallest size: its worst)
@pytest.mark.parametrize("W,H,kw,kh,bound", [(100, 100, 7, 7, 2.69e-7), (309, 152, 157, 7, 2.82e-7), (640, 480, 31, 33, 2.70e-7),
                                             (850, 850, 65, 65, 3.05e-7), (1024, 1024, 129, 129, 2.94e-7)])
def test_convolution(W, H, kw, kh, bound):
    import ghostlight_gb300 as gl
    img = [_noise(i, H, W) for i in range(3)]
    k = np.random.default_rng(kw).standard_normal((kh, kw)).astype(np.float32)
    plan = gl.ConvPlan(W, H, k)
    out = [torch.empty_like(i) for i in img]
    plan.execute(img, out)
    s = (H + kh - 1, W + kw - 1)
    K = torch.fft.rfft2(torch.from_numpy(k).cuda().double(), s=s)
    for i, o in zip(img, out):
        want = torch.fft.irfft2(torch.fft.rfft2(i.double(), s=s) * K, s=s)[kh // 2:kh // 2 + H, kw // 2:kw // 2 + W]
        assert _off(o, want) < bound
    plan.close()


def test_sprite_kernels_follow_each_other():
    """Bakes and autocorrelations without a wait between them (their launches are set
    up early) and in a graph, against the same with waits: equal bit for bit but for
    the energy's last bits (its FP64 sum has no fixed order)."""
    from ghostlight_gb300.starburst import SpritePlan
    spec = np.array([[450.0, 0.2, 0.3, 0.5], [550.0, 0.4, 0.5, 0.1], [650.0, 0.6, 0.1, 0.0]], np.float32)
    for N, ds in [(512, 64), (1024, 2), (2048, 4)]:
        plan = SpritePlan(N, spec)
        grids = [_noise(N + i, N, N).abs() for i in range(2)]
        lags = [torch.empty((65, 65), device="cuda") for _ in range(2)]
        want = []
        for g, l in zip(grids, lags):
            plan.bake(g, ds)
            torch.cuda.synchronize()
            want.append(plan.read()[:2])
            plan.autocorr(g, 32, l)
            torch.cuda.synchronize()
            want[-1] += (l.clone(),)

        def chain():
            got = []
            for g, l in zip(grids, lags):
                l.fill_(7.0)
                plan.autocorr(g, 32, l)
                plan.bake(g, ds)
                got.append(plan.read()[:2] + (l.clone(),))
            return got

        for _ in range(5):
            for a, b in zip(chain(), want):
                assert torch.equal(a[0], b[0])
                for x, y in zip(a[1:], b[1:]):
                    assert float((x - y).abs().max()) <= 2.0 ** -22 * float(y.abs().max())
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.graph(graph, stream=side):
            plan.bake(grids[0], ds)
            plan.autocorr(grids[1], 32, lags[1])
        lags[1].fill_(7.0)
        graph.replay()
        torch.cuda.synchronize()
        assert float((lags[1] - want[1][2]).abs().max()) <= 2.0 ** -22 * float(want[1][2].abs().max())
        plan.close()
