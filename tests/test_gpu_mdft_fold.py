"""The folded matrix-DFT products: reduction centres anywhere on the operand,
reduction lengths that end inside a pipeline step, and output windows at any
alignment, against a float64 evaluation of the unfolded sums."""
import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# split BF16 carries 16 bits per operand (2^-17 each) and drops lo x lo; TF32
# 11 bits, three products deep; FP32 the rounding of sums of a few hundred terms
TOL = {"split_bf16": 1e-4, "tf32": 2e-2, "fp32": 1e-5}


def _want(A, K, sx, sy, cx, cy, w, cj, box):
    n = A.shape[0]
    j = np.arange(n) - cj
    out = np.zeros((3, K[1], K[0]))
    for l in range(len(sx)):
        def mat(rows, s, c):
            m = np.exp(-2j * np.pi * s * np.outer(np.arange(rows) - c, j))
            return m * np.sinc(s * j)[None, :] if box else m
        E = mat(K[1], sy[l], cy) @ (A.astype(np.float64) @ mat(K[0], sx[l], cx).T)
        out += w[l].astype(np.float64)[:, None, None] * (E.real if box else np.abs(E) ** 2)
    return out


@pytest.mark.parametrize("form", ["split_bf16", "tf32", "fp32"])
@pytest.mark.parametrize("box,n,cj", [(False, 128, 63.5), (False, 256, 100.0), (False, 128, 0.0), (True, 128, 50.0),
                                      (True, 256, 127.5), (True, 128, 128.0)])
def test_reduction_centres(form, box, n, cj):
    import ghostlight_gb300 as gl
    r = np.random.default_rng(n + int(2 * cj))
    A = r.random((n, n)).astype(np.float32)
    K, L = (256, 128), 2
    sx, sy = np.array([0.9, 0.7]) / 256, np.array([0.8, 0.6]) / 128
    w = r.random((L, 3)).astype(np.float32)
    plan = gl.MdftPlan(n, K, sx, sy, w, form, center_x=120.3, center_y=70.7, box=box, red_center=cj)
    out = [torch.empty((K[1], K[0]), device="cuda") for _ in range(3)]
    want = _want(A, K, sx, sy, 120.3, 70.7, w, cj, box)
    for tile in (128, 64):
        plan.set_launch(0, tile)
        plan.execute(torch.from_numpy(A).cuda(), *out)
        assert plan.status() == 0
        assert rel_l2(torch.stack(out).cpu().numpy().astype(np.float64), want) < TOL[form]


@pytest.mark.parametrize("form", ["split_bf16", "fp32"])
@pytest.mark.parametrize("W,H,x0,y0,ww,wh", [(300, 200, 4, 3, 128, 128), (301, 200, 5, 0, 127, 97), (300, 160, 1, 2, 33, 5),
                                             (304, 200, 8, 1, 126, 100)])
def test_windows(form, W, H, x0, y0, ww, wh):
    """A window's pixels are the plan's own, added into the planes; nothing
    outside it is touched."""
    import ghostlight_gb300 as gl
    n = 128
    A = torch.from_numpy(np.random.default_rng(3).random((n, n)).astype(np.float32)).cuda()
    w = np.array([[1.0, 0.5, 0.25]], np.float32)
    plan = gl.MdftPlan(n, (128, 128), [1 / 128.0], [1 / 128.0], w, form, center_x=60.2, center_y=61.9)
    full = [torch.empty((128, 128), device="cuda") for _ in range(3)]
    plan.execute(A, *full)
    out = [torch.ones((H, W), device="cuda") for _ in range(3)]
    plan.execute_window(A, *out, x0, y0, ww, wh)
    for f, o in zip(full, out):
        want = torch.ones((H, W), device="cuda")
        want[y0:y0 + wh, x0:x0 + ww] += f[:wh, :ww]
        assert torch.equal(o, want)          # one wavelength: one addition per pixel
