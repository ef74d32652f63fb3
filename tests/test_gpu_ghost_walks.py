"""Which walk a plan takes, the pair-by-pair queue's wavelength splits, and what the
trace counter counts."""
import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _plan(lens, pairs, sources=1, spectral=4, grid=40, size=(200, 150), half=(15.0, 11.0), **kw):
    import ghostlight_gb300 as gl
    src = np.array([[0.05 + 0.02 * i, 0.02, 1.0, 0.8, 0.6] for i in range(sources)], np.float32)
    spec, corr = gl.spectral_table(spectral)
    return gl.GhostRenderPlan(lens, np.array(pairs, np.int32), np.ones(len(pairs), np.float32), src,
                              [gl.pupil_grid(lens, grid)], None, spec, corr, size[0], size[1], half[0], half[1], 1000.0, **kw)


def _render(plan):
    out = [torch.empty((plan.height, plan.width), device="cuda") for _ in range(3)]
    plan.execute(*out)
    torch.cuda.synchronize()
    return torch.stack(out).cpu().numpy()


def _lens(off=None):
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    lens = gl.OpticalSystem(P.double_gauss_12(seed=1))
    if off is not None:
        lens.surfaces[off].is_active = False
    return lens


@pytest.mark.parametrize("name,grid,spectral,sources,adaptive", [
    ("double_gauss_12", 8, 31, 1, False), ("wide_angle_24", 33, 5, 2, False), ("wide_angle_24", 48, 16, 1, True),
    ("anamorphic_18", 24, 8, 3, False)])
def test_plans_share_legs(name, grid, spectral, sources, adaptive):
    """The default queue walks the tree: a task is one wavelength, so splits, which
    are for the other walk, change nothing."""
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    src = np.array([[0.15 + 0.02 * i, 0.01 * i, 1.0, 0.8, 0.6] for i in range(sources)], np.float32)
    cfg = gl.FlareConfig(ray_grid=grid, spectral_samples=spectral, min_ghost_intensity=1e-7, adaptive_grids=adaptive)
    plan = gl.prepare_ghost_render(gl.OpticalSystem(getattr(P, name)()), src, 200, 150, cfg, 15.0, 11.0)
    assert plan.walk_tasks > 0 and plan.walk_tasks % spectral == 0
    assert plan.persistent_ctas <= plan.walk_tasks


def test_who_traces_pair_by_pair():
    lens = _lens()
    assert _plan(lens, [(2, 8)]).walk_tasks > 0
    assert _plan(lens, [(2, 8)], plain_per_pair=True).walk_tasks == 0
    off = _lens(3)
    assert _plan(off, [(2, 8), (4, 8)]).walk_tasks > 0
    p = _plan(off, [(2, 8), (3, 8)], cull_dead_pairs=True, grid=160)
    assert p.walk_tasks == 0 and p.probe_tasks == 0
    assert _plan(_lens(), [(2, 8), (4, 8)], cull_dead_pairs=True, grid=160).probe_tasks > 0


@pytest.mark.parametrize("ctas", [0, 4])
def test_queue_splits_pair_by_pair(ctas):
    """A plan with a pair that turns at an inactive surface: the queue and the probe
    take their wavelengths in one to 31 ranges."""
    off = 5
    lens = _lens(off)
    n = len(lens.surfaces)
    pairs = [(a, b) for b in range(n) for a in range(b) if off not in (a, b)] + [(off, n - 1)]
    plan = _plan(lens, pairs, spectral=31, grid=160, size=(96, 72), half=(1.2, 0.9), cull_dead_pairs=True)
    assert plan.walk_tasks == 0 and plan.probe_tasks == 0
    kept, imgs = {}, {}
    for chunks in (31, 1, 4, 8, 2):
        plan.set_launch(0, ctas, chunks)
        imgs[chunks] = _render(plan)
        kept[chunks] = plan.pair_hits() > 0
    assert 0 < kept[31].sum() < len(pairs) and imgs[31].sum() > 0
    for chunks in (1, 4, 8, 2):
        np.testing.assert_array_equal(kept[chunks], kept[31])
        assert rel_l2(imgs[chunks], imgs[31]) < 1e-5


def test_counter_of_the_probe():
    """No pair ever lands: every probe ray of every pair at every wavelength is
    traced, by either walk."""
    n = len(_lens().surfaces)
    pairs = [(a, b) for b in range(2, n) for a in range(b) if 5 not in (a, b)]
    kw = dict(spectral=5, grid=160, sources=2, size=(64, 48), half=(1e-7, 1e-7), cull_dead_pairs=True)
    legs = _plan(_lens(5), pairs, **kw)
    single = _plan(_lens(5), pairs + [(5, n - 1)], **kw)
    assert legs.probe_tasks > 0 and single.probe_tasks == 0
    _render(legs)
    _render(single)
    assert not legs.pair_hits().any()
    per_pair = legs.traced_split()[1] // len(pairs)
    assert legs.traced_split() == (0, per_pair * len(pairs))
    assert single.traced_split() == (0, per_pair * (len(pairs) + 1))
