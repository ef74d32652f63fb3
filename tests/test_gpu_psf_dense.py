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
