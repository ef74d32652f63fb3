"""The tree walk of the batched render against the pair-by-pair walk: same rays,
same image to the order of its additions."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _compare(lens, src, cfg, pairs=None, size=(200, 150)):
    import ghostlight_gb300 as gl
    w, h = size
    if pairs is None:
        plan = gl.prepare_ghost_render(lens, src, w, h, cfg, 15.0, 11.0)
    else:
        grid = gl.pupil_grid(lens, cfg.ray_grid)
        spec, corr = gl.spectral_table(cfg.spectral_samples)
        plan = gl.GhostRenderPlan(lens, pairs, np.ones(len(pairs), np.float32), src, [grid], None, spec, corr, w, h, 15.0,
                                  11.0, 1000.0)

    def render():
        out = [torch.empty((h, w), device="cuda") for _ in range(3)]
        plan.execute(*out)
        return torch.stack(out).double(), plan.traced_split()[0]

    got, rays = render()
    plan.set_launch(2, 0, 1)             # one-shot CTAs: pair by pair
    want, rays1 = render()
    assert rays == rays1 and float(want.sum()) > 0
    # float32 sums of a pixel's rays in another order: a few thousand terms
    assert float((got - want).norm() / want.norm()) < 1e-5


@pytest.mark.parametrize("lens,grid,spectral,sources,adaptive", [
    ("double_gauss_12", 8, 31, 1, False), ("double_gauss_12", 16, 3, 1, False), ("wide_angle_24", 33, 5, 2, False),
    ("wide_angle_24", 48, 16, 1, True), ("anamorphic_18", 24, 8, 3, False), ("double_gauss_12", 96, 31, 1, False)])
def test_tree_equals_pair_by_pair(lens, grid, spectral, sources, adaptive):
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    src = np.array([[0.15 + 0.02 * i, 0.01 * i, 1.0, 0.8, 0.6] for i in range(sources)], np.float32)
    cfg = gl.FlareConfig(ray_grid=grid, spectral_samples=spectral, min_ghost_intensity=1e-7, adaptive_grids=adaptive)
    _compare(gl.OpticalSystem(getattr(P, lens)()), src, cfg)


# neighbouring surfaces, the first and the last, one b, distinct b, an unsorted
# list with a pair twice, and a pair that turns at an inactive surface (pair by
# pair in both)
@pytest.mark.parametrize("pairs,off", [([(0, 1)], None), ([(0, 12)], None), ([(11, 12), (0, 12), (5, 12)], None),
                                       ([(1, 3), (4, 6), (7, 9)], None), ([(5, 9), (0, 4), (5, 9), (2, 9), (3, 4)], None),
                                       ([(2, 8), (3, 8), (1, 4)], 5), ([(2, 8), (3, 8)], 3)])
def test_pair_lists(pairs, off):
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    lens = gl.OpticalSystem(P.double_gauss_12(seed=1))
    if off is not None:
        lens.surfaces[off].is_active = False
    src = np.array([[0.05, 0.02, 1.0, 0.8, 0.6]], np.float32)
    _compare(lens, src, gl.FlareConfig(ray_grid=40, spectral_samples=4), pairs=np.array(pairs, np.int32))


def test_focused_ghost_sums_in_the_warp():
    """A sensor of metres: every landing of a warp falls into one footprint, which
    the tree walk sums first.  One pair, 208 samples, 3 wavelengths: at most 624
    float32 additions to a pixel in either order, 624 x 2^-24 apart at most."""
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    lens = gl.OpticalSystem(P.double_gauss_12(seed=1))
    src = np.array([[0.02, 0.01, 1.0, 0.8, 0.6]], np.float32)
    spec, corr = gl.spectral_table(3)
    plan = gl.GhostRenderPlan(lens, [(2, 9)], [1.0], src, [gl.pupil_grid(lens, 16)], None, spec, corr, 7, 5, 4000.0, 4000.0,
                              1000.0)

    def render():
        out = [torch.empty((5, 7), device="cuda") for _ in range(3)]
        plan.execute(*out)
        return torch.stack(out).double()

    got = render()
    plan.set_launch(2, 0, 1)
    want = render()
    assert float(want.sum()) > 0
    assert float((got - want).abs().max()) <= 624 * 2.0 ** -24 * float(want.max())


@pytest.mark.parametrize("lens,sources,spectral,off", [("wide_angle_24", 1, 31, 7), ("wide_angle_24", 3, 4, 7),
                                                        ("anamorphic_18", 2, 9, 6), ("anamorphic_18", 1, 5, 6)])
def test_probe_culls_the_same_pairs(lens, sources, spectral, off):
    """A plan with a pair that turns at an inactive surface is probed pair by pair:
    the other pairs must come out the same as from the tree."""
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    lens = gl.OpticalSystem(getattr(P, lens)())
    lens.surfaces[off].is_active = False
    n = len(lens.surfaces)
    pairs = [(a, b) for b in range(n) for a in range(b) if off not in (a, b)]
    src = np.array([[0.3 + 0.02 * i, 0.2 * i, 1.0, 0.8, 0.6] for i in range(sources)], np.float32)
    spec, corr = gl.spectral_table(spectral)

    def culled(pairs):
        plan = gl.GhostRenderPlan(lens, pairs, np.ones(len(pairs), np.float32), src, [gl.pupil_grid(lens, 160)], None, spec,
                                  corr, 64, 48, 1.2, 0.9, 1000.0, cull_dead_pairs=True)
        out = [torch.empty((48, 64), device="cuda") for _ in range(3)]
        plan.execute(*out)
        return [int(h) > 0 for h in plan.pair_hits()], out

    got, image = culled(pairs)
    want, _ = culled(pairs + [(off, n - 1)])
    assert got[:len(pairs)] == want[:len(pairs)]
    assert 0 < sum(got[:len(pairs)]) < len(pairs)
    assert all(bool(torch.isfinite(c).all()) for c in image)
