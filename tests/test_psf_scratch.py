"""Admission of served PSF atlases: the scratch of a wide splat's landings counts
against the HBM budget, and is what a request gives up when the budget is short."""
import pytest

from ghostlight_gb300.serve import FlareRequest, FlareServer, psf_request_bytes


def _request(extent, rid=0, grid=8, tile=64):
    return FlareRequest(lens_id=0, width=grid * tile, height=grid * tile, n_spec=16, ray_grid=64, field_deg=0.0, rid=rid,
                        kind="psf", psf_grid=grid, psf_tile=tile, psf_extent_mm=extent)


@pytest.mark.parametrize("extent,wide", [(0.05, True), (0.2, True), (0.4, False)])
def test_landings_are_counted(extent, wide):
    total, landing = psf_request_bytes(_request(extent))
    planes = 2 * 3 * 4 * 512 * 512
    assert total - landing >= planes
    if not wide:
        assert landing == 0
        return
    # 64 sources x 16 wavelengths x the pupil's disc of 64^2 samples, 16 bytes each
    assert 64 * 16 * int(0.78 * 64 * 64) * 16 <= landing <= 64 << 20


class _Exec:
    """Executor that takes estimates only."""

    def __init__(self):
        self.started = []

    def estimate(self, req):
        req.device_bytes, req.landing_bytes = psf_request_bytes(req)

    def start(self, req):
        self.started.append(req)
        return req

    def done(self, run):
        return False


def test_budget():
    total, landing = psf_request_bytes(_request(0.05))
    assert landing > 0
    # room for one and a half: the second waits
    ex = _Exec()
    srv = FlareServer({}, budget_bytes=total * 3 // 2, executor=ex)
    for i in range(2):
        srv.submit(_request(0.05, rid=i))
    srv.step()
    assert [r.rid for r in ex.started] == [0] and srv.sched.used <= srv.sched.budget
    assert ex.started[0].landing_bytes == landing
    # less than one: admitted with as much as fits
    for short in (1 << 20, landing):
        ex = _Exec()
        srv = FlareServer({}, budget_bytes=total - short, executor=ex)
        srv.submit(_request(0.05))
        srv.step()
        r = ex.started[0]
        assert r.landing_bytes == landing - short and r.device_bytes == srv.sched.budget
    # less than the planes: rejected, as before
    srv = FlareServer({}, budget_bytes=total - landing - 1, executor=_Exec())
    srv.submit(_request(0.05))
    assert len(srv.rejected) == 1
