"""The wavelength split that a plan picks for itself: one task per wavelength
on the smallest plans, the default on large ones; every split traces the same
rays and gives the same image to the order of its additions."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,spectral,sources,adaptive", [(8, 31, 1, False), (16, 3, 1, False), (33, 5, 2, False),
                                                            (48, 16, 1, True), (96, 31, 1, False)])
def test_picked_split_equals_one_task(grid, spectral, sources, adaptive):
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    lens = gl.OpticalSystem(P.double_gauss_12(seed=1))
    src = np.array([[0.15 + 0.02 * i, 0.01 * i, 1.0, 0.8, 0.6] for i in range(sources)], np.float32)
    cfg = gl.FlareConfig(ray_grid=grid, spectral_samples=spectral, min_ghost_intensity=1e-7, adaptive_grids=adaptive)
    plan = gl.prepare_ghost_render(lens, src, 200, 150, cfg, 15.0, 11.0)

    def render():
        out = [torch.empty((150, 200), device="cuda") for _ in range(3)]
        plan.execute(*out)
        return torch.stack(out).double(), plan.traced_split()[0]

    got, rays = render()
    plan.set_launch(0, 0, 1)
    want, rays1 = render()
    assert rays == rays1 and float(want.sum()) > 0
    # float32 sums of a pixel's rays in another order: a few thousand terms
    assert float((got - want).norm() / want.norm()) < 1e-5
