"""The wavelength bake's box sums over the thread's rows, lanes, warps and the
second pass, against the float64 restatement."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import sprite_oracle as SO

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# rows per thread 1 (256) and 4; box sums within the rows, across
# lanes, across warps (above the rows) and above 32 (second pass); more
# wavelengths than one staging (64).  1e-4: a float32 sample position at 1000
# texels is known to 6e-5 of a texel.
@pytest.mark.parametrize("N,ds,ns", [(256, 1, 5), (256, 4, 5), (256, 32, 70), (512, 4, 5), (512, 8, 5), (512, 64, 3),
                                     (1024, 8, 3), (1024, 16, 4), (1024, 128, 3)])
def test_box_sums(N, ds, ns):
    from ghostlight_gb300.starburst import SpritePlan
    lam = np.linspace(380.0, 760.0, ns, dtype=np.float32)
    spec = np.stack([lam, np.sin(lam) ** 2 / ns, np.cos(lam) ** 2 / ns, np.full(ns, 1.0 / ns)], 1).astype(np.float32)
    y, x = np.mgrid[0:N, 0:N] - (N - 1) / 2
    pupil = ((np.hypot(x, y) < 0.11 * N) & (x > -0.08 * N)).astype(np.float32)
    plan = SpritePlan(N, spec)
    plan.bake(torch.from_numpy(pupil).cuda(), ds)
    _, spr, _ = plan.read()
    got = spr.cpu().numpy()
    plan.close()
    assert got.shape == (N // ds, N // ds, 3)
    assert rel_l2(got, SO.sprite(pupil, spec, ds)) < 1e-4
