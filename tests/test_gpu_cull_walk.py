"""The culler's one-walk probes against the float oracle's filter: set, order,
boosts and footprints bit for bit, from a two-surface lens to the longest
walks, with no silhouette, one, several, tilted ones and inactive surfaces."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _lens(kind):
    from ghostlight_gb300 import prescriptions as P
    if kind == "single":
        s = P.double_gauss_12(seed=1)[:2]
        P.finalize_z(s)
        return s
    if kind == "long":                              # 57 surfaces, one stop
        s = []
        for k in range(4):
            s += [x for x in P.double_gauss_12(seed=k + 1) if not x.is_stop or k == 0]
        s += P.double_gauss_12(seed=9)[:8]
        for x in s:
            x.semi_aperture = 40.0 if not x.is_stop else x.semi_aperture
            x.thickness = min(x.thickness, 2.0)
        P.finalize_z(s)
        return s
    s = P.random_lens(seed=5, n_surfaces=int(kind.split("_")[1]))
    if "round" in kind:
        for x in s:
            x.aperture_shape, x.aperture_blades = 0, 0
    if "many" in kind:                              # a second and a third silhouette, one of them tilted
        for i in (0, len(s) - 2):
            s[i].aperture_shape, s[i].aperture_blades, s[i].aperture_rotation_rad = 1, 7, 0.3
        c, t = np.cos(0.01), np.sin(0.01)
        for i, v in enumerate((1, 0, 0, 0, c, -t, 0, t, c)):
            s[0].rot[i] = float(v)
    if "off" in kind:
        s[3].is_active = 0
    return s


@pytest.mark.parametrize("kind", ["single", "random_8", "random_30", "random_20_round", "random_20_many", "random_12_off", "long"])
def test_filter_matches_oracle(kind):
    import ghostlight_gb300 as gl
    from ghostlight_gb300.flare import filter_ghosts_device
    from oracle import oracle as O
    recs = _lens(kind)
    lens = gl.OpticalSystem.from_records(recs)
    for thr in (0.0, 1e-7, 1e-5):
        r = filter_ghosts_device(lens, 18.0, 12.0, gl.FlareConfig(min_ghost_intensity=thr))
        pairs, boosts, fp = O.filter_pairs(lens.records(), 18.0, 12.0, thr, footprint=True)
        np.testing.assert_array_equal(r.pairs, pairs)
        # the oracle's cosf / atan2f may round a weight's last place otherwise; boxes are IEEE-exact
        np.testing.assert_allclose(r.boosts, boosts, rtol=1e-5)
        np.testing.assert_allclose(r.footprint_mm, fp, rtol=1e-5)
