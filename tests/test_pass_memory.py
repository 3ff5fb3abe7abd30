"""The buffers of passes of several steps in a server's memory accounting."""
import pytest

from conftest import same
from lbc_gb300 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fits", [True, False])
def test_budget_holds_the_buffers_of_passes(fits):
    """A request whose batch steps in passes holds two more population buffers:
    they count as bytes in use while it is active, and a budget without room for
    them leaves passes out; the result is the same."""
    from lbc_gb300 import F32_SHIFTED, GpuServer, GpuSolver
    case, st = cases.cavity_moving_wall(2100, 0.1, 300.0)
    pops = 9 * 4 * 2112 * 2100                # one buffer: rows padded to 64 nodes
    est = 2 * pops + 60 * case.nodes          # the rest: fields, staging, flags
    srv = GpuServer(est + 2 * pops + (1 << 20) if fits else est + pops, 64, 120)
    rid = srv.submit(case, st, 360, F32_SHIFTED)
    most, room, before = 0, 1 << 62, srv.available()
    while srv.poll() > 0:
        most, room = max(most, srv.stats()["bytes"]), min(room, srv.available())
    assert srv.stats()["bytes"] == 0
    if fits:
        assert most >= 4 * pops
        assert before - room >= 4 * pops
    else:
        assert 2 * pops < most <= est
        assert before - room < 4 * pops
    got = srv.fetch(rid)
    s = GpuSolver(case, F32_SHIFTED)
    s.set_state(st)
    s.run(360)
    want = s.get_fields()
    for a, b in zip((got["rho"], got["u"], got["v"]), want):
        assert same(a, b)
    s.close()
    srv.release(rid)
    srv.close()
