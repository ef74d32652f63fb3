"""The setup's beams, traced in groups of rays side by side, against the float
oracle's ray-by-ray trace: equal bit for bit.  37 rays a beam, so the last
group is a partial one; lenses that mix plain spheres and planes with the
surfaces that are still traced one ray at a time."""
import ctypes as C

import numpy as np
import pytest

f = np.float32


def _lens(kind):
    import ghostlight_gb300 as gl
    from ghostlight_gb300 import prescriptions as P
    base = {"aspheric": P.wide_angle_24}.get(kind, P.double_gauss_12)
    lens = gl.OpticalSystem(base())
    stop = next(s for s in lens.surfaces if s.is_stop)
    if kind == "plane":
        lens.surfaces[3].radius = 0.0
    elif kind == "inactive":
        lens.surfaces[2].is_active = False
    elif kind == "aspect":
        lens.surfaces[1].aperture_aspect = 1.3
    elif kind == "triangle":
        stop.aperture_shape, stop.aperture_blades, stop.aperture_rotation_rad = 1, 3, 0.3
    elif kind == "round":
        stop.aperture_shape = 0
    return lens


@pytest.mark.parametrize("kind", ["common", "aspheric", "plane", "inactive", "aspect", "triangle", "round"])
def test_beam_equals_ray_by_ray(kind):
    from ghostlight_gb300 import _native
    from ghostlight_gb300._abi import gl_psf_cell
    from oracle import oracle as O
    lens = _lens(kind)
    recs, arr = lens.records(), lens.to_array()
    src = np.zeros((5, 7), f)
    src[:, :2] = [[0, 0], [0.12, -0.05], [-0.2, 0.1], [0.33, 0.28], [0.6, 0.0]]
    cells = (gl_psf_cell * len(src))()
    lib = _native.load()
    _native.check(lib.gl_psf_prepass(arr, len(arr), src.ctypes.data_as(C.POINTER(C.c_float)), len(src), 0, cells), "prepass")
    R = f(recs[0].semi_aperture)
    g = [f(-1.0) + (f(i) + f(0.5)) * (f(2.0) / f(7)) for i in range(7)]
    uv = [(u, v) for v in g for u in g if u * u + v * v <= f(1.0)]
    assert len(uv) == 37
    lit = 0
    for k, (ax, ay) in enumerate(src[:, :2]):
        bx, by = f(np.tan(ax)), f(np.tan(ay))
        d = np.array([bx, by, 1.0], f)
        d = (d * (f(1.0) / f(np.sqrt(f(f(d[0] * d[0]) + f(d[1] * d[1])) + f(1.0))))).astype(f)
        rays = np.array([[u * R - f(20.0) * bx, v * R - f(20.0) * by, f(recs[0].z) - f(20.0), *d, f(587.56)] for u, v in uv], f)
        res = O.trace(recs, -1, -1, rays, fp64=False)
        ok = (res[:, 4] == 0) & np.isfinite(res[:, 0]) & np.isfinite(res[:, 1])
        if not ok.any():
            continue                    # dark, or found through the axial window
        lit += 1
        sx = sy = f(0.0)
        for x, y in res[ok][:, :2]:
            sx, sy = f(sx + f(x)), f(sy + f(y))
        n = f(int(ok.sum()))
        assert (f(cells[k].chief_x_mm), f(cells[k].chief_y_mm)) == (f(sx / n), f(sy / n))
        assert f(cells[k].pupil_fraction) == f(n / f(len(uv)))
    assert lit >= 2
