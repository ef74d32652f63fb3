"""A matrix-DFT whose pupil lies in the memory of its output planes: the pupil is
read before the planes are zeroed, so the result is that of separate buffers.
One wavelength: one addition to a pixel, equal bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,box", [("split_bf16", False), ("split_bf16", True), ("tf32", False), ("fp32", False),
                                      ("fp32", True)])
@pytest.mark.parametrize("n,K", [(512, 1024), (128, 256)])
def test_pupil_in_a_plane(form, box, n, K):
    import ghostlight_gb300 as gl
    r = np.random.default_rng(n)
    A = torch.from_numpy(r.random((n, n)).astype(np.float32)).cuda()
    plan = gl.MdftPlan(n, K, [0.9 / K], [0.8 / K], r.random((1, 3)).astype(np.float32), form, center_x=K / 2 - 0.7,
                       center_y=K / 2 + 0.3, box=box)
    want = torch.empty((3, K, K), device="cuda")
    plan.execute(A, *want)
    # at the first plane's start, across the first two, at the last plane's end
    for start in (0, K * K - 100, 3 * K * K - n * n):
        buf = torch.zeros(3 * K * K, device="cuda")
        pupil = buf[start:start + n * n].view(n, n)
        pupil.copy_(A)
        got = buf.view(3, K, K)
        plan.execute(pupil, *got)
        assert plan.status() == 0
        assert torch.equal(got, want)
