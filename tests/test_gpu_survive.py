"""The survivor centre and envelope made on the device against the same
construction on host arrays with the batched device trace: the same launches
through the same trace, so only a launch within rounding of an edge (of an
aperture, or of the stop's silhouette) may fall on the other side."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _lens(kind):
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    lens = gl.OpticalSystem((P.wide_angle_24 if kind == "wide" else P.anamorphic_18 if kind == "anamorphic"
                             else P.double_gauss_12)())
    stop = next(s for s in lens.surfaces if s.is_stop)
    if kind == "round":
        stop.aperture_shape = 0
    elif kind == "triangle":
        stop.aperture_shape, stop.aperture_blades, stop.aperture_rotation_rad = 1, 3, 0.3
    return lens


@pytest.mark.parametrize("kind,field,me", [("polygon", (0.1, 0.05), 64), ("polygon", (0.0, -0.17), 33), ("round", (0.15, 0.0), 16),
                                           ("triangle", (-0.1, 0.08), 129), ("wide", (0.3, 0.1), 64),
                                           ("anamorphic", (0.05, -0.1), 48), ("polygon", (1.4, 0.0), 16)])
def test_device_equals_host_arrays(kind, field, me):
    from ghostlight_gb300 import starburst as S
    lens = _lens(kind)
    ep = float(lens.calibration().entrance_pupil_semi_x)

    def survives(x, y, z, d):
        return S._survives_device(lens, x, y, z, d)

    got, want = S.survivor_center(lens, *field), S.survivor_center(lens, *field, survives=survives)
    assert got[2] == want[2]
    # 81 x 81 cells over 2.2 front radii and a launch in 64 of one: a launch that
    # falls on the other side moves the mean of n cells by at most reach / (64 n)
    reach = 1.2 * lens.surfaces[0].semi_aperture + 40.0
    assert max(abs(got[0] - want[0]), abs(got[1] - want[1])) <= 4 * reach / (64 * 100)
    env = S.survivor_envelope(lens, ep, ep, want[0], want[1], *field, me)
    ref = S.survivor_envelope(lens, ep, ep, want[0], want[1], *field, me, survives=survives)
    assert env.shape == ref.shape == (me, me) and env.dtype == np.float32
    # cells apart: at most 2 in 1000 (those beside an edge that passes a launch
    # within rounding), nearly all by one launch in 100
    off = np.abs(env - ref)
    assert (off > 0).mean() <= 2e-3
    assert not (off > 0).any() or np.median(off[off > 0]) <= 0.02
    assert env.min() >= 0.0 and env.max() <= 1.0
