"""The one-kernel steps end at each row of a series.  Once the call that asked for
it has ended -- by its steps, or by its time -- the kernels of the systems that
go on are as long as without it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402


def _arm(b, i, steps, series=None, every=0, limit=-1.0):
    b.engine.call_begin_many([b.states[i].slot], steps, [1e-4], limit, series=series, series_every=every)


def _run(b, steps):
    before = b.engine.launches()
    b.run(steps)
    return b.engine.launches() - before


@pytest.mark.parametrize("ctas", [0, -1])
def test_rows_stop_with_their_call(ctas):
    b = Batch([W.make_system(f"s{i}", 2, 60, 10, 40.0, seed=i) for i in range(2)], precision="fp64", ctas_per_sm=ctas)
    b.set_adaptive(True)
    buf = torch.zeros((1, 40, 5), dtype=torch.float64, device=b.device)
    _arm(b, 0, 31, buf, 3)
    _arm(b, 1, 1000)
    queued = _run(b, 1000)
    # the check, ten rows of three steps, 512 and 458 steps, each with the series kernel
    assert ctas < 0 or queued == 1 + 2 * 12
    sts = b.statuses()
    assert [s["steps_done"] for s in sts] == [31, 1000] and sts[0]["series_rows"] == 10
    np.testing.assert_array_equal(buf[0, :10, 0].cpu().numpy(), np.arange(3, 31, 3))
    # by its time: known to have ended once its status has been read
    _arm(b, 0, -1, buf, 3, limit=1e-3)
    _arm(b, 1, 200)
    _run(b, 200)
    sts = b.statuses()
    assert not sts[0]["active"] and sts[0]["series_rows"] == sts[0]["steps_done"] // 3
    _arm(b, 1, 1000)
    assert ctas < 0 or _run(b, 1000) == 1 + 2 * 2
    b.close()
