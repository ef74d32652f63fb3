"""Operands that start off the boundaries of the kernels' wide accesses: a
contiguous view at any float offset gives what the aligned tensor gives."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _at_offset(a, off):
    """A contiguous copy of `a` whose first element lies `off` floats past a
    256-byte boundary."""
    buf = torch.zeros(a.numel() + 64, dtype=torch.float32, device="cuda")
    v = buf[off:off + a.numel()].view(a.shape)
    v.copy_(a)
    assert v.is_contiguous() and v.data_ptr() % 16 == 4 * off % 16
    return v


# ping-pong and in-place column transforms
@pytest.mark.parametrize("N", [256, 1024, 2048])
def test_sprite_pupil(N):
    from ghostlight_gb300.starburst import SpritePlan
    r = np.random.default_rng(N)
    y, x = np.mgrid[0:N, 0:N] - (N - 1) / 2
    pupil = torch.from_numpy(((np.hypot(x, y) < 0.15 * N) * r.random((N, N))).astype(np.float32)).cuda()
    spec = np.array([[450.0, 0.2, 0.3, 0.5], [550.0, 0.4, 0.5, 0.1], [650.0, 0.6, 0.1, 0.0]], np.float32)
    plan = SpritePlan(N, spec)

    def run(p):
        plan.bake(p, 4)
        psf, sprite, energy = plan.read()
        lags = torch.empty((65, 65), device="cuda")
        plan.autocorr(p, 31, lags)
        return psf, sprite, lags, energy

    want = run(pupil)
    assert want[3] > 0
    for off in (1, 2, 3):
        got = run(_at_offset(pupil, off))
        assert torch.equal(got[0], want[0])
        # the energy's FP64 sum has no fixed order: its last bits may turn a scale's rounding
        assert got[3] == pytest.approx(want[3], rel=1e-12)
        for a, b in zip(got[1:3], want[1:3]):
            assert float((a - b).abs().max()) <= 2.0 ** -22 * float(b.abs().max())
    plan.close()
