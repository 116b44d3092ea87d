"""Contexts that share the device (``ctas_per_sm`` > 0) sum the pair forces of
2D mixed batches in the pair kernel; a context alone lets its stages walk the
lists.  Both run the same sums in the same order: every bit is the same."""
import copy

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200.batch import Batch  # noqa: E402
from gliding_collective_rotation_b200.workloads import config3  # noqa: E402


@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("block", [64, 128])
def test_pair_kernel_and_own_walk_agree(order, block):
    # 5 systems of over 1000 beads: more than the 16 tiles that would step in
    # one kernel in a context of several, and tiles with a remainder
    specs = sorted(config3(n_systems=64, param_seed=11), key=lambda s: s.n)[:5]
    assert sum(-(-s.n // block) for s in specs) > 16
    out = []
    for ctas in (-1, 1, 9):
        b = Batch([copy.deepcopy(s) for s in specs], precision="mixed", ctas_per_sm=ctas, block_beads=block,
                  srk_order=order)
        b.set_adaptive(True)
        b.begin(30)
        b.run(30)
        st = b.statuses()
        assert all(s["flags"] == 0 and s["steps_done"] == 30 for s in st)
        out.append(([x.pos.cpu().numpy() for x in b.states], [s["dt"] for s in st]))
        b.close()
    for pos, dts in out[1:]:
        assert dts == out[0][1]
        for p, q in zip(pos, out[0][0]):
            np.testing.assert_array_equal(p, q)
