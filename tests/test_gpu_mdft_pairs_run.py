"""That pairs of CTAs are taken where they should be, and several wavelengths
through them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _plan(n, K, L, form="split_bf16", **kw):
    import ghostlight_gb300 as gl
    r = np.random.default_rng(n + K[0])
    return gl.MdftPlan(n, K, np.linspace(0.6, 0.9, L) / K[0], np.linspace(0.5, 0.8, L) / K[1],
                       r.random((L, 3)).astype(np.float32), form, center_x=K[0] / 2 - 0.7, center_y=K[1] / 2 + 0.3, **kw)


# which of the two products run in pairs: the first from reductions of 16 stages on
# (a pupil of 2048), the second from 8 (512)
@pytest.mark.parametrize("n,K,L,want", [(512, (2560, 2560), 1, (False, True)), (2048, (1536, 1536), 1, (True, True)),
                                        (2048, (1536, 256), 1, (True, False)), (512, (2560, 2432), 1, (False, False)),
                                        (512, (512, 256), 1, (False, False)), (512, (1024, 1024), 7, (False, True)),
                                        (1024, (768, 1280), 5, (False, True))])
def test_where_pairs_run(n, K, L, want):
    plan = _plan(n, K, L)
    got = plan.cta_pairs()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert tuple(p > 0 for p in got) == want and max(got) <= sms // 2
    plan.set_launch(1)
    assert plan.cta_pairs() == (0, 0)
    plan.set_launch(5)
    assert tuple(p > 0 for p in plan.cta_pairs()) == want and max(plan.cta_pairs()) <= 2
    plan.set_launch(0, 64)
    assert plan.cta_pairs()[1] == 0
    plan.close()


def test_other_forms_run_single_ctas():
    for form, kw in [("tf32", {}), ("split_bf16", {"box": True}), ("fp32", {})]:
        assert _plan(512, (2560, 2560), 1, form, **kw).cta_pairs() == (0, 0)


@pytest.mark.parametrize("n,K,L", [(512, (1024, 1024), 7), (1024, (768, 1280), 5)])
def test_several_wavelengths(n, K, L):
    """The same products wavelength by wavelength, one CTA at a time: their additions
    to a pixel come in any order, L x 2^-24 apart at most."""
    A = torch.from_numpy(np.random.default_rng(L).random((n, n)).astype(np.float32)).cuda()
    plan = _plan(n, K, L)
    assert plan.cta_pairs()[1] > 0
    out = torch.empty((3, K[1], K[0]), device="cuda")
    plan.execute(A, *out)
    assert plan.status() == 0
    plan.set_launch(1)
    want = torch.zeros_like(out)
    for l in range(L):
        plan.set_lambda_range(l, l + 1)
        plan.execute(A, *want, accumulate=True)
    assert float(want.max()) > 0
    assert bool(((out - want).abs() <= L * 2.0 ** -24 * want.abs()).all())
    plan.close()
