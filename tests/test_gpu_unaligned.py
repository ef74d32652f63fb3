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


# field and pixel form, both tiles of the second product, a pair of CTAs (2560)
@pytest.mark.parametrize("form,K,box", [("split_bf16", 256, False), ("split_bf16", 256, True), ("split_bf16", 2560, False),
                                        ("tf32", 256, False), ("tf32", 256, True), ("fp32", 256, False), ("fp32", 256, True)])
def test_mdft_planes(form, K, box):
    """One wavelength: one addition to a pixel, so equal bit for bit.  Planes that
    start at different offsets, too, and the pupil at one."""
    import ghostlight_gb300 as gl
    n = 512 if K == 2560 else 128
    r = np.random.default_rng(K)
    A = torch.from_numpy(r.random((n, n)).astype(np.float32)).cuda()
    plan = gl.MdftPlan(n, K, [0.9 / K], [0.8 / K], r.random((1, 3)).astype(np.float32), form, center_x=K / 2 - 0.7,
                       center_y=K / 2 + 0.3, box=box)
    for tile in (128,) if K == 2560 else (128, 64):
        plan.set_launch(0, tile)
        want = [torch.empty((K, K), device="cuda") for _ in range(3)]
        plan.execute(A, *want)
        assert float(want[0].abs().max()) > 0
        for offs in [(1, 1, 1), (2, 2, 2), (3, 3, 3), (0, 1, 0), (0, 0, 2)]:
            got = [_at_offset(torch.full((K, K), 7.0), o) for o in offs]
            plan.execute(_at_offset(A, offs[1]), *got)
            assert plan.status() == 0
            assert all(torch.equal(a, b) for a, b in zip(got, want))
        frame = [_at_offset(torch.zeros((K + 3, K + 8)), o) for o in (3, 0, 1)]
        plan.execute_window(A, *frame, 4, 2, K - 5, K - 9)
        for f, w in zip(frame, want):
            assert torch.equal(f[2:2 + K - 9, 4:4 + K - 5], w[:K - 9, :K - 5])
