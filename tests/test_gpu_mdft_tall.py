"""The FP32 matrix-DFT's tall tiles (enough of them for half of the SMs) against
a float64 evaluation of the sums: whole planes, and windows that end inside a
tile at aligned and unaligned places."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_mdft_fold import TOL, _want

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [False, True])
@pytest.mark.parametrize("K,L", [((640, 512), 4), ((256, 1280), 3), ((1024, 128), 31)])
def test_tall_tiles(K, L, box):
    import ghostlight_gb300 as gl
    n = 128
    r = np.random.default_rng(K[0] + L)
    A = r.random((n, n)).astype(np.float32)
    sx, sy = np.linspace(0.6, 0.9, L) / K[0], np.linspace(0.5, 0.8, L) / K[1]
    w = r.random((L, 3)).astype(np.float32)
    cx, cy = K[0] / 2 - 0.7, K[1] / 2 + 0.3
    plan = gl.MdftPlan(n, K, sx, sy, w, "fp32", center_x=cx, center_y=cy, box=box, red_center=70.5)
    want = _want(A, K, sx, sy, cx, cy, w, 70.5, box)
    op = torch.from_numpy(A).cuda()
    out = [torch.empty((K[1], K[0]), device="cuda") for _ in range(3)]
    plan.execute(op, *out)
    assert rel_l2(torch.stack(out).cpu().numpy().astype(np.float64), want) < TOL["fp32"]
    for x0, width in [(8, K[0] + 16), (5, K[0] + 11)]:
        ww, wh = K[0] - 37, K[1] - 70
        frame = [torch.zeros((K[1] + 3, width), device="cuda") for _ in range(3)]
        plan.execute_window(op, *frame, x0, 2, ww, wh)
        got = torch.stack(frame).cpu().numpy().astype(np.float64)
        assert rel_l2(got[:, 2:2 + wh, x0:x0 + ww], want[:, :wh, :ww]) < TOL["fp32"]
        got[:, 2:2 + wh, x0:x0 + ww] = 0.0
        assert not got.any()
