"""A served system that stopped in the middle of a step leaves with its flag,
relaxing or not, and is not carried into a regrown context; the others finish."""
import pytest

from gliding_collective_rotation_b200._lib import FLAG_CELL_OVERFLOW, FLAG_WAIT_EXPIRED
from tests.test_serve_host import FakeEngine, FakeServer, _requests


class TornEngine(FakeEngine):
    """The first run stops slot 0 in the middle of a step and overflows slot 1."""

    torn = False

    def call_begin_many(self, slots, *a, **kw):
        assert not any(self.sys[s]["flags"] & FLAG_WAIT_EXPIRED for s in slots)  # the library refuses it
        super().call_begin_many(slots, *a, **kw)

    def run(self, n):
        super().run(n)
        if not TornEngine.torn:
            TornEngine.torn = True
            self.sys[0]["flags"] = FLAG_WAIT_EXPIRED
            self.sys[1]["flags"] = FLAG_CELL_OVERFLOW


class TornServer(FakeServer):
    def _make_engine(self):
        eng = TornEngine(self.bead_capacity, self.max_systems)
        self.engines.append(eng)
        return eng


@pytest.mark.parametrize("relax", [False, True])
def test_a_torn_system_leaves_with_its_flag(relax):
    TornEngine.torn = False
    srv = TornServer(hbm_budget=1 << 26, chunk=64)
    res = {r.id: r for r in srv.serve(_requests(3, 200, relax=relax), timeout=30)}
    assert sorted(res) == [0, 1, 2] and len(srv.engines) == 2
    assert res[0].flags == FLAG_WAIT_EXPIRED and res[0].steps < 200
    assert all(res[i].flags == 0 and res[i].steps == 200 for i in (1, 2))
