"""A wide splat's landings in several rounds over sources and wavelengths, and the
atlas without them (each ray its own taps): the same terms in another order, over
windows wider than the splat needs, tiles off the composite and dim sources too."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_rounds():
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    from ghostlight_gb300.psf_grid import psf_inputs, psf_launch
    lens = gl.OpticalSystem(P.double_gauss_12(seed=1))
    src = np.array([[0.02 * i, 0.03 * j, 1.0, 0.8, 0.6] for j in range(2) for i in range(3)], np.float32)
    cfg = gl.PSFConfig(grid_nx=3, grid_ny=2, tile_w=48, tile_h=40, tile_extent_mm=0.12, ray_grid=30, spectral_samples=7,
                       splat_sigma_um=2.0 * 120.0 / 48)
    inp = psf_inputs(src, lens, cfg)

    def run(landing_bytes):
        out = torch.zeros((3, inp["comp_h"], inp["comp_w"]), device="cuda")
        psf_launch(inp, out, torch.cuda.current_stream().cuda_stream, ordered=True, landing_bytes=landing_bytes)
        n = gl._native.last_launch_count()
        return out.double(), n

    want, n = run(None)
    assert n == 2 and float(want.max()) > 0
    one = 16 * len(inp["grid"])                 # a wavelength of a source
    # (sources, wavelengths) at a time: (1, 1), (1, 5), (1, 7), (2, 7), (6, 7)
    for k, launches in [(1, 84), (5, 24), (8, 12), (14, 6), (42, 2)]:
        got, n = run(k * one)
        assert n == launches
        assert float((got - want).norm() / want.norm()) < 1e-6
    for few in (0, one - 1):
        got, n = run(few)
        assert n == 1
        assert float((got - want).norm() / want.norm()) < 2e-5


def test_more_landings_than_the_scratch():
    """8 x 8 sources, 31 wavelengths, 64^2 samples: 6 M landings in two rounds of
    the full scratch, against the sources one by one."""
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    lens = gl.OpticalSystem(P.double_gauss_12(seed=1))
    cfg = dict(tile_w=32, tile_h=32, tile_extent_mm=0.1, ray_grid=64, spectral_samples=31, splat_sigma_um=6.0)
    src = np.array([[0.01 * i, 0.01 * j, 1.0, 0.8, 0.6] for j in range(8) for i in range(8)], np.float32)
    out = gl.render_psf(src, lens, gl.PSFConfig(grid_nx=8, grid_ny=8, **cfg))
    assert gl._native.last_launch_count() == 4
    for i in (0, 9, 40, 41, 42, 63):
        one = gl.render_psf(src[i:i + 1], lens, gl.PSFConfig(grid_nx=1, grid_ny=1, **cfg))
        for k in ("r", "g", "b"):
            y, x = i // 8 * 32, i % 8 * 32
            a, b = out[k][y:y + 32, x:x + 32].double(), one[k].double()
            assert float(b.max()) > 0 and float((a - b).norm() / b.norm()) < 1e-6


def _pair(inp):
    """(with landings, taps) as float64 planes."""
    from ghostlight_gb300.psf_grid import psf_launch
    got = []
    for landing_bytes in (None, 0):
        out = torch.zeros((3, inp["comp_h"], inp["comp_w"]), device="cuda")
        psf_launch(inp, out, torch.cuda.current_stream().cuda_stream, ordered=True, landing_bytes=landing_bytes)
        torch.cuda.synchronize()
        got.append((out.double(), __import__("ghostlight_gb300")._native.last_launch_count()))
    assert got[0][1] == 2 and got[1][1] == 1          # landings and tiles; taps
    return got[0][0], got[1][0]


# radii of the splat (2.5 sigma: with and without taps below 1e-6) and beyond it;
# float32 sums of some thousand terms in other orders, and taps within rounding of
# the line on the other side of it, 1e-6 of a splat each
@pytest.mark.parametrize("sigma,radius", [(0.85, 3), (1.1, 3), (1.25, 4), (1.62, 5), (5.12, 13), (0.3, 16), (0.9, 14), (1.5, 10),
                                          (3.0, 16), (7.0, 4)])
@pytest.mark.parametrize("mono", [False, True])
def test_windows_equal_taps(sigma, radius, mono):
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    from ghostlight_gb300.psf_grid import psf_inputs
    lens = gl.OpticalSystem(P.double_gauss_12(seed=1))
    src = np.array([[0.02 * i, 0.01 * i, 1.0, 0.8, -0.2 * i] for i in range(4)], np.float32)
    cfg = gl.PSFConfig(grid_nx=2, grid_ny=2, tile_w=43, tile_h=30, tile_extent_mm=0.1, ray_grid=24, spectral_samples=5,
                       monochromatic=mono)
    inp = psf_inputs(src, lens, cfg)
    inp["sigma"], inp["radius"] = sigma, radius
    inp["sources"][1].tile_x0, inp["sources"][1].tile_y0 = 60, -7          # partly off the composite
    a, b = _pair(inp)
    assert float(b.abs().max()) > 0
    assert float((a - b).norm() / b.norm()) < 2e-6


def test_dim_sources_equal_taps():
    """Colours around which a ray's share in a plane passes 1e-14, the least that a
    plane takes: in all planes, in some, in none."""
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    from ghostlight_gb300.psf_grid import psf_inputs
    s = P.double_gauss_12(seed=1)
    # weights over five decades: an attenuator's Gaussian
    s[2].coating_model, s[2].gauss_sigma, s[2].gauss_background, s[2].gauss_peak = 4, 4.0, 1e-5, 1.0
    lens = gl.OpticalSystem(s)
    src = np.array([[0.0, 0.0, 1e-9, 1e-11, 1e-13], [0.02, 0.0, 1e-8, 1e-8, 1e-8], [0.0, 0.02, 1e-15, 1e-16, 0.0],
                    [0.02, 0.02, 1e-10, 0.0, 1e-3]], np.float32)
    cfg = gl.PSFConfig(grid_nx=2, grid_ny=2, tile_w=40, tile_h=40, tile_extent_mm=0.1, ray_grid=32, spectral_samples=9)
    inp = psf_inputs(src, lens, cfg)
    inp["sigma"], inp["radius"] = 2.0, 5
    a, b = _pair(inp)
    for k in range(3):
        for y in (0, 40):
            for x in (0, 40):
                u, v = a[k, y:y + 40, x:x + 40], b[k, y:y + 40, x:x + 40]
                assert bool((v != 0).any()) == bool((u != 0).any())
                assert float((u - v).norm()) <= 2e-6 * float(v.norm())
    assert float(b[0].abs().max()) > 0 and not b[:, 40:, :40].any()
