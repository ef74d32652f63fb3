"""The FP32 matrix-DFT repeats bit for bit, however its wavelengths are split over
CTAs, and its two-level sums keep the pattern's peak."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_mdft_fold import TOL, _want

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# short tiles, tall tiles, several groups of wavelengths (1.6 M pixels, ten planes at
# a time), tiles enough without a split
@pytest.mark.parametrize("n,K,L,box", [(256, (256, 128), 31, False), (256, (512, 512), 8, False), (128, (512, 384), 8, True),
                                       (128, (1536, 1024), 31, False), (128, (2048, 1280), 3, False)])
def test_repeats(n, K, L, box):
    import ghostlight_gb300 as gl
    r = np.random.default_rng(K[0] + L)
    A = r.random((n, n)).astype(np.float32)
    sx, sy = np.linspace(0.6, 0.9, L) / K[0], np.linspace(0.5, 0.8, L) / K[1]
    w = r.random((L, 3)).astype(np.float32)
    plan = gl.MdftPlan(n, K, sx, sy, w, "fp32", center_x=K[0] / 2 - 0.7, center_y=K[1] / 2 + 0.3, box=box)
    op = torch.from_numpy(A).cuda()
    out = torch.empty((3, K[1], K[0]), device="cuda")
    plan.execute(op, *out)
    want = out.clone()
    ref = _want(A, K, sx, sy, K[0] / 2 - 0.7, K[1] / 2 + 0.3, w, 0.5 * (n - 1), box)
    assert rel_l2(want.cpu().numpy().astype(np.float64), ref) < TOL["fp32"]
    for _ in range(10):
        plan.execute(op, *out)
        assert torch.equal(out, want)
    # into a window, added to what is there, and planes that are one and the same
    for x0, width in [(8, K[0] + 16), (5, K[0] + 11)]:
        ww, wh = K[0] - 37, K[1] - 70
        frame = torch.zeros((3, K[1] + 3, width), device="cuda")
        plan.execute_window(op, *frame, x0, 2, ww, wh)
        assert torch.equal(frame[:, 2:2 + wh, x0:x0 + ww], want[:, :wh, :ww])
        frame[:, 2:2 + wh, x0:x0 + ww] = 0.0
        assert not frame.any()
    one = torch.zeros((K[1], K[0]), device="cuda")
    plan.execute(op, one, one, one, accumulate=True)
    assert float((one - want.sum(0)).abs().max()) <= 4 * 2.0 ** -24 * float(want.sum(0).abs().max())
    # part of the wavelengths, and the rest on top
    cut = L // 2
    plan.set_lambda_range(0, cut)
    plan.execute(op, *out)
    plan.set_lambda_range(cut, L)
    plan.execute(op, *out, accumulate=True)
    assert float((out - want).abs().max()) <= (L + 2) * 2.0 ** -24 * float(want.abs().max())
    plan.close()


def test_peak_of_two_level_sums():
    """At the pattern's centre every factor is 1: the pupil's sum over 256 distances
    twice, squared.  A sum of m like terms rounds to about 0.58 sqrt(m / 3) 2^-24 of
    itself (rms): 16 blocks of 16 terms, 1.3 x 2^-24 for the blocks' sum and a quarter
    of that for the blocks, doubled by the square: 1.6e-7.  256 terms in one sum:
    6.4e-7.  The bound lies between."""
    import ghostlight_gb300 as gl
    n, K = 512, 128
    plan = gl.MdftPlan(n, K, [0.9 / K], [0.8 / K], np.ones((1, 3), np.float32), "fp32", center_x=64.0, center_y=50.0)
    out = [torch.empty((K, K), device="cuda") for _ in range(3)]
    off = []
    for seed in range(32):
        A = np.random.default_rng(seed).random((n, n)).astype(np.float32)
        plan.execute(torch.from_numpy(A).cuda(), *out)
        off.append(float(out[0][50, 64]) / A.astype(np.float64).sum() ** 2 - 1.0)
    assert np.sqrt(np.mean(np.square(off))) < 3.2e-7
    plan.close()


@pytest.mark.parametrize("form", ["fp32", "split_bf16"])
def test_in_a_graph(form):
    """Captured calls, after a copy and after another kernel, and with the pupil in a
    plane (memsets between the launches): what the calls give outside the graph."""
    import ghostlight_gb300 as gl
    n, K, L = 128, 384, 1 if form == "split_bf16" else 6
    r = np.random.default_rng(5)
    A = torch.from_numpy(r.random((n, n)).astype(np.float32)).cuda()
    plan = gl.MdftPlan(n, K, np.linspace(0.6, 0.9, L) / K, np.linspace(0.5, 0.8, L) / K, r.random((L, 3)).astype(np.float32), form)
    want = torch.empty((3, K, K), device="cuda")
    plan.execute(A, *want)
    op, out, buf = torch.empty_like(A), torch.empty_like(want), torch.empty_like(want)
    inside = buf.view(-1)[K * K - 100:K * K - 100 + n * n].view(n, n)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        op.copy_(A)
        plan.execute(op, *out)
        plan.execute(op, *out, accumulate=True)
        inside.copy_(A)
        plan.execute(inside, *buf)
    for _ in range(3):
        op.zero_()
        out.fill_(3.0)
        buf.fill_(5.0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(buf, want)
        assert torch.equal(out, want + want)
    plan.close()
