"""Wide-Gaussian PSF tiles (the dense kernel) against the float-oracle restatement."""
import numpy as np
import pytest

from conftest import lens_from_pins, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# the kernel's 8 x 8 pixel blocks: whole, one row over, a tile smaller than the
# window, the largest tile (every thread one block) and one past it (the sparse
# kernel); grids below and above one CTA's samples.  2e-3: a float32 landing is
# known to about 2e-6 mm, 2e-3 px at the finest pitch here, against a splat of
# at least 1.2 px.
@pytest.mark.parametrize("tile_w,tile_h,grid,sigma_px", [(64, 64, 24, 1.2), (65, 33, 40, 2.0), (9, 8, 24, 6.0),
                                                         (128, 128, 16, 3.0), (129, 128, 16, 3.0)])
def test_psf_dense_tiles(pins, tile_w, tile_h, grid, sigma_px):
    import ghostlight_gb300 as gl
    from ghostlight_gb300.flare import pupil_grid
    from ghostlight_gb300.psf_grid import _psf_spectrum, splat_footprint
    from oracle import psf_oracle as PO
    from tests_psf_cells import cells_of
    lens = gl.OpticalSystem.from_records(lens_from_pins(pins, "cfg1_double_gauss_12"))
    cfg = gl.PSFConfig(grid_nx=2, grid_ny=2, tile_w=tile_w, tile_h=tile_h, tile_extent_mm=0.12, ray_grid=grid,
                       spectral_samples=4, splat_sigma_um=sigma_px * 120.0 / tile_w)
    src = np.array([[0.0, 0.0, 1.0, 0.8, 0.6, 0.0, 0.0], [0.08, 0.03, 0.5, 1.0, 0.7, 0.0, 0.0],
                    [-0.1, 0.06, 1.0, 1.0, 1.0, 0.0, 0.0]], np.float32)
    out = gl.render_psf(src, lens, cfg)
    got = np.stack([out[k].cpu().numpy() for k in ("r", "g", "b")]).astype(np.float64)
    mm_pp = float(np.float32(cfg.tile_extent_mm) / np.float32(cfg.tile_w))
    sigma, radius = splat_footprint(cfg.splat_sigma_um, mm_pp)
    want = PO.render(lens.records(), cells_of(lens, src, 0), src[:, 2:5], pupil_grid(lens, grid), _psf_spectrum(cfg),
                     tile_w, tile_h, 2, 2 * tile_w, 2 * tile_h, mm_pp, False, sigma, radius)
    assert want.sum() > 0
    assert rel_l2(got, want) < 2e-3


def test_wavelengths_split_into_uneven_parts(pins):
    """25 sources of 13 blocks: the landings' 31 wavelengths go in parts of 3, the
    last one shorter.  The same atlas without the splat's Gaussian being dense
    (bilinear) carries the same energy into each tile: the Gaussian is normalised
    and 2 px wide here, and the landings stay clear of the 64 px tiles' borders.
    Float32 sums of ~80,000 weights: 80,000 x 2^-24 apart at most, and the
    Gaussian's taps below 1e-6 of its sum are left out (25 x 25 of them at most)."""
    import ghostlight_gb300 as gl
    lens = gl.OpticalSystem.from_records(lens_from_pins(pins, "cfg1_double_gauss_12"))
    src = np.array([[0.02 * i, 0.02 * j, 1.0, 0.8, 0.6, 0.0, 0.0] for j in range(5) for i in range(5)], np.float32)
    energy = []
    for sigma_um in (0.0, 25.0):
        cfg = gl.PSFConfig(grid_nx=5, grid_ny=5, tile_w=64, tile_h=64, tile_extent_mm=0.8, ray_grid=64, spectral_samples=31,
                           splat_sigma_um=sigma_um)
        out = gl.render_psf(src, lens, cfg)
        a = np.stack([out[k].cpu().numpy() for k in ("r", "g", "b")]).astype(np.float64)
        energy.append(a.reshape(3, 5, 64, 5, 64).sum((2, 4)))
    assert energy[0].min() > 0
    assert np.abs(energy[1] / energy[0] - 1.0).max() <= 80000 * 2.0 ** -24 + 625e-6
