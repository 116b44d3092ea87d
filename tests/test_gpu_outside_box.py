"""Positions that a caller has not wrapped into the box: in a box of 3 or 4
cells a side the first lists hold every pair, as with the wrapped positions, and
the first forces are the same.

Tolerance: a separation of about 1 from coordinates of up to 5.5 carries a few
1e-16, the WCA force takes it times 14, and a bead sums at most 26 of them:
1e-11 of the largest force is far above that and far below any missing pair.
"""
import copy

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402


def _first_step(spec, ctas):
    b = Batch([copy.deepcopy(spec)], precision="fp64", ctas_per_sm=ctas, list_depth=128)
    b.begin(1, dt=1e-9)
    b.run(1)
    st = b.statuses()[0]
    assert st["flags"] == 0 and st["steps_done"] == 1 and st["list_builds"] == 1
    counts, partners, _, total = b.engine.neighbour_list(0)
    out = counts.cpu().numpy(), partners.cpu().numpy(), total, b.states[0].forces.cpu().numpy()
    b.close()
    return out


@pytest.mark.parametrize("ctas", [0, -1])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("L", [4.0, 5.4])
def test_lists_and_forces_of_unwrapped_positions(L, dim, ctas):
    side = int(L / 0.9)
    spec = W.make_system("box", dim, side ** dim, 1, L, seed=1)
    rs = np.random.default_rng(5)
    grid = np.stack(np.meshgrid(*[np.arange(side)] * dim, indexing="ij"), -1).reshape(-1, dim)
    spec.pos[:] = np.mod((grid + 0.5) * (L / side) + rs.uniform(-0.05, 0.05, grid.shape), L)
    want = _first_step(spec, ctas)
    assert want[2] > 2 * dim * len(grid) - 1  # every lattice neighbour within the list radius
    centred = copy.deepcopy(spec)
    centred.pos[centred.pos >= L / 2] -= L
    got = _first_step(centred, ctas)
    assert got[2] == want[2]
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
    assert np.abs(got[3] - want[3]).max() <= 1e-11 * np.abs(want[3]).max()
