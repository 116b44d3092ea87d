"""The per-system work of a step: over the slots in use, by one CTA for each 1024
of them.  More systems than that step as they do in smaller batches, bit for
bit, and slots that hold no system cost nothing.

The time of 16,384 slots with one system in use is 1.0 of that of 1 slot when only
slots in use are visited, and was 2.6 when all were: 1.6 tells them apart."""
import copy
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402
from gliding_collective_rotation_b200.engine import Engine, SystemState  # noqa: E402


def _specs(n):
    out = []
    for i in range(n):
        s = W.make_system(f"s{i}", 2, 1 + i % 3, 4 + i % 5, 9.0 + i % 4, seed=i, T=0.2)
        s.params.max_dist_per_step = s.relax_mdps
        out.append(s)
    return out


def _run(specs, steps, ctas):
    b = Batch([copy.deepcopy(s) for s in specs], precision="fp64", ctas_per_sm=ctas)
    b.engine.call_begin_many([s.slot for s in b.states], steps, 1e-4)
    b.run(30)
    sts = b.statuses()
    out = [s.pos.cpu().numpy() for s in b.states], [(s["steps_done"], s["dt"], s["list_builds"]) for s in sts]
    assert all(s["flags"] == 0 for s in sts)
    b.close()
    return out


@pytest.mark.parametrize("n", [1024, 1025, 2100])
def test_many_systems_step_as_in_smaller_batches(n):
    specs = _specs(n)
    steps = [30 if i % 7 else 11 for i in range(n)]  # some systems end their call before the others
    pos, sts = _run(specs, steps, 0)
    for lo in range(0, n, 500):
        p, s = _run(specs[lo:lo + 500], steps[lo:lo + 500], -1)
        assert s == sts[lo:lo + 500]
        for x, y in zip(p, pos[lo:lo + 500]):
            np.testing.assert_array_equal(x, y)


def _us_per_step(capacity):
    eng = Engine(2, "mixed", bead_capacity=1 << 16, system_capacity=capacity, block_beads=128)
    s = W.make_system("s", 2, 200, 10, 60.0, seed=3)
    s.params.max_dist_per_step = s.relax_mdps
    st = SystemState.from_host(s.pos, s.tangent, s.chain_id, s.rest_lengths, s.params, "mixed")
    eng.admit(st)
    best = 1e9
    for k in range(8):
        eng.call_begin(st.slot, 500, 1e-5 if k == 0 else 0.0)
        torch.cuda.synchronize()
        t = time.perf_counter()
        eng.run(500)
        torch.cuda.synchronize()
        best = min(best, (time.perf_counter() - t) / 500 * 1e6)
    eng.close()
    return best


def test_empty_slots_cost_nothing():
    assert _us_per_step(16384) < 1.6 * _us_per_step(1)


@pytest.mark.parametrize("n,one_kernel", [(128, True), (129, False)])
def test_one_kernel_while_each_slot_has_a_thread(n, one_kernel):
    b = Batch(_specs(n), precision="fp64")  # blocks of 128 threads
    b.begin(10, dt=1e-4)
    before = b.engine.launches()
    b.run(10)
    assert (b.engine.launches() - before == 2) == one_kernel
    b.close()
