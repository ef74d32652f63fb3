"""The split-BF16 field form's error against float64 about different reduction
centres: at most that of the unfolded sums (measured, mean of four pupils and
scales, and a tenth above it), and less about the pupil's middle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _error(n, kind, rc):
    import ghostlight_gb300 as gl
    K, L, e = (384, 256), 2, []
    for seed in range(4):
        r = np.random.default_rng([n, seed])
        y, x = np.mgrid[0:n, 0:n] - (n - 1) / 2
        A = ((np.hypot(x, y) < 0.4 * n) * 1.0) if kind == "disc" else r.uniform(-0.1, 1.0, (n, n))
        A = torch.from_numpy(A.astype(np.float32)).cuda()
        sx, sy = r.uniform(0.3, 1, L) / K[0], r.uniform(0.3, 1, L) / K[1]
        w, cx, cy = r.uniform(0, 1, (L, 3)).astype(np.float32), r.uniform(100, 300), r.uniform(80, 180)
        plan = gl.MdftPlan(n, K, sx, sy, w, "split_bf16", center_x=cx, center_y=cy, red_center=rc)
        out = torch.empty((3, K[1], K[0]), device="cuda")
        plan.execute(A, *out)
        j = torch.arange(n, device="cuda", dtype=torch.float64) - rc
        want = torch.zeros_like(out, dtype=torch.float64)
        for l in range(L):
            def mat(rows, s, c):
                p = -2 * np.pi * s * torch.outer(torch.arange(rows, device="cuda", dtype=torch.float64) - c, j)
                return torch.complex(torch.cos(p), torch.sin(p))
            E = mat(K[1], sy[l], cy) @ (A.to(torch.complex128) @ mat(K[0], sx[l], cx).T)
            for c in range(3):
                want[c] += float(w[l, c]) * E.abs() ** 2
        e.append(float((out.double() - want).norm() / want.norm()))
        plan.close()
    return np.mean(e)


@pytest.mark.parametrize("n,kind,rc,unfolded", [(128, "noise", 12.5, 1.67e-6), (128, "noise", 95.5, 1.46e-6), (256, "disc", 25.5, 2.09e-6),
                                                (256, "disc", 102.0, 2.09e-6), (256, "disc", 191.0, 2.27e-6),
                                                (512, "disc", 204.5, 3.95e-6)])
def test_off_the_middle(n, kind, rc, unfolded):
    assert _error(n, kind, rc) < 1.1 * unfolded


@pytest.mark.parametrize("n,kind,unfolded", [(128, "disc", 1.70e-6), (128, "noise", 1.48e-6), (256, "disc", 2.05e-6), (512, "noise", 8.25e-6)])
def test_about_the_middle(n, kind, unfolded):
    assert _error(n, kind, 0.5 * (n - 1)) < unfolded
