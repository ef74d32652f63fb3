"""The split-BF16 matrix-DFT in pairs of CTAs (one product of 256 rows, half of
B in each) against the same plan one CTA at a time (a grid of one has no room
for a pair): one wavelength and planes that start at zero, so every pixel takes
one addition, and the products are summed in the same order: equal bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# pairs in step 2 (400 units of 8 stages, and of 12 with a partial last one), in
# both steps, in step 1 only, row blocks that do not come in pairs, too few units
@pytest.mark.parametrize("n,K,cj", [(512, (2560, 2560), 255.5), (512, (2560, 2560), 179.0), (2048, (1536, 1536), 1023.5),
                                    (2048, (1536, 256), 1023.5), (512, (2560, 2432), 255.5), (512, (512, 256), 255.5)])
def test_pairs_equal_single_ctas(n, K, cj):
    import ghostlight_gb300 as gl
    r = np.random.default_rng(n + K[0])
    A = torch.from_numpy(r.random((n, n)).astype(np.float32)).cuda()
    plan = gl.MdftPlan(n, K, np.array([0.9 / K[0]]), np.array([0.8 / K[1]]), r.random((1, 3)).astype(np.float32), "split_bf16",
                       center_x=K[0] / 2 - 0.7, center_y=K[1] / 2 + 0.3, red_center=cj)

    def run(ctas, tile):
        plan.set_launch(ctas, tile)
        out = [torch.empty((K[1], K[0]), device="cuda") for _ in range(3)]
        plan.execute(A, *out)
        assert plan.status() == 0
        return torch.stack(out)

    want = run(1, 128)
    assert float(want.abs().max()) > 0
    for ctas, tile in [(0, 128), (0, 64), (2, 128), (5, 64), (7, 128)]:
        assert torch.equal(run(ctas, tile), want)
