"""Values at the edges of what the wide-Gaussian PSF tiles take: weights below zero
(an attenuator may have them), a source colour that is not a number."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SRC = np.array([[0.0, 0.0, 1.0, 0.8, 0.6, 0.0, 0.0], [0.08, 0.03, 0.5, 1.0, 0.7, 0.0, 0.0]], np.float32)


# a splat of 2 px (wide) and one of 0.5 px (narrow)
@pytest.mark.parametrize("sigma_px", [2.0, 0.5])
def test_negative_weights(sigma_px):
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    cfg = gl.PSFConfig(grid_nx=2, grid_ny=1, tile_extent_mm=0.12, ray_grid=40, spectral_samples=4,
                       splat_sigma_um=sigma_px * 120.0 / 64)
    got = []
    for bg in (0.5, -0.5):
        s = P.double_gauss_12(seed=1)
        s[4].coating_model, s[4].gauss_sigma, s[4].gauss_background, s[4].gauss_peak = 4, 0.0, bg, 0.0
        out = gl.render_psf(SRC, gl.OpticalSystem(s), cfg)
        got.append(torch.stack([out[k] for k in ("r", "g", "b")]).double())
    assert float(got[0].max()) > 0 and float(got[1].min()) < 0
    # the same terms with the other sign, their additions in another order
    assert float((got[0] + got[1]).norm() / got[0].norm()) < 1e-5


def test_colour_not_a_number():
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    from ghostlight_gb300.psf_grid import psf_inputs, psf_launch
    lens = gl.OpticalSystem(P.double_gauss_12(seed=1))
    for sigma_px in (2.0, 0.5):
        cfg = gl.PSFConfig(grid_nx=2, grid_ny=1, tile_extent_mm=0.12, ray_grid=24, spectral_samples=4,
                           splat_sigma_um=sigma_px * 120.0 / 64)
        inp = psf_inputs(SRC, lens, cfg)
        planes = []
        for r in (1.0, float("nan")):
            inp["sources"][0].r = r
            out = torch.zeros((3, inp["comp_h"], inp["comp_w"]), device="cuda")
            psf_launch(inp, out, torch.cuda.current_stream().cuda_stream)
            planes.append(out)
        good, bad = planes
        assert float(good[0, :, :64].max()) > 0
        assert not bad[0, :, :64].any()                       # the tap kernel's answer: nothing added
        for a, b in ((bad[0, :, 64:], good[0, :, 64:]), (bad[1], good[1]), (bad[2], good[2])):
            assert float((a - b).double().norm() / b.double().norm()) < 1e-5
