"""One FP64 step of small systems whose chains cross the edges of warps (32
beads) and tiles (64 or 128 beads), on the GPU against the oracle.

The stage kernels take a bead's neighbours along the chain by warp shuffles
and compute three bonds and two bends beside each warp again; the lists of
these systems are empty, short (one flattened round) and long (walked rows).
Positions are of order 10, so one rounding of a step is about 2e-15; 1e-13
leaves fifty of them and is far below any missing or doubled term (a bond or
bend moves a bead by more than 1e-6).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200.batch import Batch  # noqa: E402
from gliding_collective_rotation_b200.engine import SystemParams  # noqa: E402
from gliding_collective_rotation_b200.engine import wca_params as make_WCA_params  # noqa: E402
from gliding_collective_rotation_b200.workloads import LJ_CUTOFF, SystemSpec  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests.golden_io import min_image  # noqa: E402


def _spec(dim, n, length, cutoff, seed=5):
    rs = np.random.default_rng([seed, dim, n, length])
    L = 24.0
    pos, tan, chain = [], [], []
    for c, begin in enumerate(range(0, n, length)):
        m = min(length, n - begin)
        m = m if m > 1 else 0  # a single bead left over joins the chain before
        y, z = 0.6 + 1.05 * (c % 21), 0.6 + 1.05 * (c // 21)
        for j in range(m):
            x = [0.5 + 0.5 * j + 8.0 * (c // 21) + rs.normal(0, 0.01), y + 0.05 * np.sin(0.9 * j) + rs.normal(0, 0.005), z]
            pos.append(np.mod(x[:dim], L))
            tan.append(np.eye(dim)[0])
            chain.append(c)
    while len(pos) < n:
        pos.append(np.mod(pos[-1] + 0.5 * np.eye(dim)[0], L))
        tan.append(np.eye(dim)[0])
        chain.append(chain[-1])
    params = SystemParams(L=L, spring_params=np.array([100.0, 20.0, 0.0, 0.0, 1.0, 0.1]),
                          wca_params=make_WCA_params(1.0, 0.5, 0.0, cutoff),
                          active_params=np.array([1.0, 0.0, 0.2 if dim == 2 else 0.0]), D=0.01, Dr=0.0075,
                          radius=1.0, n_nearby=4, dtmax=1e-3, max_dist_per_step=0.0125, seed=seed)
    return SystemSpec("edges", dim, np.array(pos), np.array(tan), np.array(chain), np.full(chain[-1] + 1, 0.5),
                      params, 1e-3, 0.0125)


@pytest.mark.parametrize("dim,cutoff", [(2, 1.0), (2, LJ_CUTOFF), (3, LJ_CUTOFF)])
@pytest.mark.parametrize("n,length", [(2, 2), (31, 4), (32, 32), (33, 33), (63, 5), (64, 31), (65, 16), (127, 3),
                                      (128, 34), (129, 32), (130, 7), (385, 40)])
def test_a_step_at_warp_and_tile_edges(dim, cutoff, n, length):
    spec = _spec(dim, n, length, cutoff)
    p = spec.params
    ng = max(1, int(p.L / (2.0 * max(1.0, p.wca_params[3]))))
    o = O.OracleSystem(spec.pos, spec.tangent, spec.chain_id, spec.rest_lengths, p.L, p.spring_params, p.wca_params,
                       p.active_params, p.D, p.Dr, p.radius, p.n_nearby, ng, nbor_depth=256)
    o.build_lists(grid_window=max(1, int(np.ceil(p.wca_params[3] / (p.L / ng)))))
    res = o.run(1, dt=1e-4, dtmax=p.dtmax, max_dist_per_step=p.max_dist_per_step, noise_mode=O.NOISE_PHILOX,
                seed=p.seed)
    for mode, block in ((0, 128), (1, 64)):
        b = Batch([spec], precision="fp64", pair_mode=mode, block_beads=block, list_depth=128)
        b.begin(1, dt=1e-4)
        b.run(1)
        st = b.statuses()[0]
        assert st["steps_done"] == 1 and st["flags"] == 0
        assert abs(st["dt"] - res["dt"]) <= 1e-11 * res["dt"]
        err = np.max(np.abs(min_image(b.states[0].pos.cpu().numpy() - o.pos, p.L)))
        assert err < 1e-13, (mode, err)
        b.close()
