"""The library counts the step kernels it queues, whichever route a batch takes:
one kernel for up to 512 steps, or graphs of steps_per_graph steps of so many
kernels each, with the run-start check before."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402


def _queued(b, steps):
    b.begin(steps)
    before = b.engine.launches()
    b.run(steps)
    return b.engine.launches() - before


@pytest.mark.parametrize("kw,a_step", [
    (dict(), 0),
    (dict(ctas_per_sm=-1), 10),  # the stages walk the lists
    (dict(ctas_per_sm=-1, precision="fp64"), 12),  # two pair kernels
    (dict(pair_mode=2, precision="fp64"), 14),  # and two sorts
    (dict(ctas_per_sm=-1, srk_order=4), 18)])
def test_kernels_queued(kw, a_step):
    kw = dict(dict(precision="mixed"), **kw)
    b = Batch([W.make_system("s", 2, 300, 10, 60.0, seed=1)], **kw)
    b.set_adaptive(True)
    for steps in (1, 10, 1000):
        graphs = -(-steps // 10)
        assert _queued(b, steps) == (2 + 10 * graphs * a_step if a_step else 1 + -(-steps // 512))
    if kw.get("srk_order", 2) == 2:  # launched one by one, whatever the route
        b.begin(3)
        before = b.engine.launches()
        b.engine.profile_steps(3)
        assert b.engine.launches() - before == 2 + 3 * (a_step or 10)
    b.close()
