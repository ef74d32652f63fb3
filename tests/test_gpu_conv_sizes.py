"""The convolution's transform lengths: every radix alone and in turn, odd
lengths (no middle bin), odd heights (a row without a partner), ping-pong and
in-place stages, one-point and few-point transforms, against float64."""
import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# padded lengths (P, Q): 1 x 1, 2 x 3, 4 x 8, 9 x 27, 81 x 243, 16 x 48, 128 x 162,
# 768 x 864 (one stage form each side of the line), 972 x 1024, 729 x 1458
@pytest.mark.parametrize("H,W,kh,kw", [(1, 1, 1, 1), (2, 1, 1, 3), (4, 6, 1, 3), (7, 25, 3, 3), (79, 239, 3, 5),
                                       (14, 46, 3, 3), (123, 155, 5, 7), (760, 858, 9, 7), (965, 1018, 7, 7),
                                       (721, 1450, 9, 9)])
def test_transform_lengths(H, W, kh, kw):
    import ghostlight_gb300 as gl
    r = np.random.default_rng(H * 7 + W)
    img = [torch.from_numpy(r.random((H, W)).astype(np.float32)).cuda() for _ in range(3)]
    add = [torch.from_numpy(r.random((H, W)).astype(np.float32)).cuda() for _ in range(3)]
    k = r.random((kh, kw)).astype(np.float32)
    out = [torch.empty_like(i) for i in img]
    plan = gl.ConvPlan(W, H, k)
    plan.execute(img, out, add=add)
    s = (H + kh - 1, W + kw - 1)
    K = np.fft.rfft2(k.astype(np.float64), s)
    for i, a, o in zip(img, add, out):
        full = np.fft.irfft2(np.fft.rfft2((i + a).cpu().numpy().astype(np.float64), s) * K, s)
        want = full[kh // 2:kh // 2 + H, kw // 2:kw // 2 + W]
        # float32 rounding of sums of a few dozen products through ~20 butterfly levels
        assert rel_l2(o.cpu().numpy().astype(np.float64), want) < 1e-6
