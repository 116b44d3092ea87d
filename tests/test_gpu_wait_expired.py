"""A wait of the one-kernel steps that runs out: the kernel ends, the systems
that were stepping carry a flag of their own, and a state whose parts may be a
step apart is not stepped on."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import updates  # noqa: E402
from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200._lib import FLAG_WAIT_EXPIRED, GcrError  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402
from gliding_collective_rotation_b200.engine import Engine  # noqa: E402
from tests.golden_io import load  # noqa: E402
from tests.gpu_helpers import pop_from_golden, set_config, status_from_row  # noqa: E402


def _specs():
    # 40 tiles of 64 beads: clusters that meet at the counter in global memory
    return [W.make_system("large", 2, 250, 10, 60.0, seed=1), W.make_system("done", 2, 4, 10, 20.0, seed=2)]


def test_the_wait_runs_out(monkeypatch):
    monkeypatch.setenv("GCR_TEAM_POLLS", "1")
    b = Batch(_specs(), precision="fp64", block_beads=64)
    monkeypatch.delenv("GCR_TEAM_POLLS")
    b.set_adaptive(True)
    slots = [s.slot for s in b.states]
    b.engine.call_begin_many(slots, [500, 0], [1e-4, 1e-4])
    b.run(500)
    large, done = b.statuses()
    assert large["flags"] == FLAG_WAIT_EXPIRED and large["steps_done"] < 500
    assert done["flags"] == 0  # it was not stepping
    with pytest.raises(GcrError, match="middle of a step"):
        b.begin(10)
    with pytest.raises(GcrError, match="middle of a step"):
        b.engine.call_begin(slots[0], 10, 1e-4)
    with pytest.raises(RuntimeError, match="middle of a step"):
        b.regrow()
    b.engine.call_begin(slots[1], 10, 1e-4)
    # admitted again with a whole state, the system steps
    spec, st = _specs()[0], b.states[0]
    b.engine.evict(slots[0])
    st.pos.copy_(torch.from_numpy(spec.pos))
    st.tangent.copy_(torch.from_numpy(spec.tangent))
    b.engine.admit(st)
    b.engine.call_begin(st.slot, 0, 1e-4)
    assert b.engine.status(st.slot)["flags"] == 0
    b.close()
    # the context is as usable as the device: with the usual bound it runs through
    b = Batch(_specs(), precision="fp64", block_beads=64)
    b.set_adaptive(True)
    sts = b.run_checked(100)
    assert all(s["flags"] == 0 and s["steps_done"] == 100 for s in sts)
    b.close()


def test_the_drop_in_hands_no_torn_state_back(monkeypatch):
    d, s = load("config1")
    set_config(s)
    sim = {"gpu_precision": "fp64", "gpu_noise": "philox", "seed": 5, "save_state_every": -1.0}

    def call(pop):
        st = status_from_row(d["status_before"][0])
        st.next_output_step = st.stepnum + 20
        updates.SRK2_force_calc([pop], st, sim)
        return st

    pop, fresh = pop_from_golden(d, s), pop_from_golden(d, s)
    before = [np.array(pop.pos), np.array(pop.tangent_list), np.array(pop.forces)]
    real = Engine.status
    monkeypatch.setattr(Engine, "status", lambda self, slot: dict(real(self, slot), flags=FLAG_WAIT_EXPIRED))
    with pytest.raises(GcrError, match="as before the call"):
        call(pop)
    for x, y in zip(before, (pop.pos, pop.tangent_list, pop.forces)):
        np.testing.assert_array_equal(x, y)
    monkeypatch.undo()
    call(pop)
    call(fresh)
    np.testing.assert_array_equal(pop.pos, fresh.pos)
