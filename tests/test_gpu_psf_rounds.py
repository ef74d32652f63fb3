"""A wide splat's landings in several rounds over sources and wavelengths, and the
atlas without them (each ray its own taps): the same terms in another order.
Taps below 1e-6 of their splat are in the former only: at most 1e-5 of it at 2 px."""
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
