"""Rigid rods step to the same bits launch by launch and in one kernel, alone and
in a batch too large for one kernel, in both precisions and SRK orders."""
import copy

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402


def _step(specs, precision, order, ctas):
    b = Batch([copy.deepcopy(s) for s in specs], precision=precision, srk_order=order, ctas_per_sm=ctas)
    b.set_adaptive(True)
    b.begin(5, dt=1e-4)
    b.run(5)
    torch.cuda.synchronize()
    n = specs[0].n
    out = [b.big[k][:n].cpu().numpy() for k in ("pos", "pos1", "forces", "tangent")]
    b.close()
    return out


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("T,clen", [(0.0, 10), (0.05, 3), (0.5, 33)])
def test_rods_alone_and_in_a_batch(precision, order, dim, T, clen):
    rods = W.make_system("rods", dim, 60, clen, 90.0 if dim == 2 else 40.0, seed=clen, T=T)
    rods.params.rigid_rod = 0.5
    # 614 tiles more: launches
    many = W.make_system("many", dim, 7850, 10, 400.0 if dim == 2 else 80.0, seed=1)
    alone = _step([rods], precision, order, 0)
    for other in (_step([rods], precision, order, -1), _step([rods, many], precision, order, 0)):
        for x, y in zip(alone, other):
            np.testing.assert_array_equal(x, y)
