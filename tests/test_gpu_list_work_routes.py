"""Small batches whose list builds are large -- a dilute box of many cells, a
population beside a much larger fixed one -- step by launches, which spread a
build over the device; in one kernel it would be the work of a few CTAs."""
import copy

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402


def _queued(specs, couple=None, **kw):
    b = Batch([copy.deepcopy(s) for s in specs], precision="fp64", **kw)
    if couple is not None:
        b.couple(*couple)
    b.set_adaptive(True)
    b.begin(10, dt=1e-5)
    before = b.engine.launches()
    b.run(10)
    queued = b.engine.launches() - before
    pos = [s.pos.cpu().numpy() for s in b.states]
    b.close()
    return queued, pos


@pytest.mark.parametrize("dim,L,one_kernel", [(2, 300.0, True), (2, 3000.0, False), (3, 60.0, True), (3, 240.0, False)])
def test_dilute_boxes(dim, L, one_kernel):
    specs = [W.make_system("s", dim, 100, 10, L, seed=3, T=1.0)]
    queued, pos = _queued(specs)
    assert (queued == 2) == one_kernel
    np.testing.assert_array_equal(pos[0], _queued(specs, ctas_per_sm=-1)[1][0])


@pytest.mark.parametrize("n_fixed,one_kernel", [(1000, True), (100000, False)])
def test_a_population_beside_a_fixed_one(n_fixed, one_kernel):
    L = max(30.0, (1.5 * n_fixed) ** 0.5)
    specs = [W.make_system("moving", 2, 20, 5, L, seed=1), W.make_system("fixed", 2, n_fixed // 5, 5, L, seed=2)]
    cross = np.zeros((2, 2, 4))
    cross[0, 1] = cross[1, 0] = specs[0].params.wca_params
    queued, pos = _queued(specs, ([0, 1], [False, True], cross))
    assert (queued == 2) == one_kernel
    np.testing.assert_array_equal(pos[0], _queued(specs, ([0, 1], [False, True], cross), ctas_per_sm=-1)[1][0])
