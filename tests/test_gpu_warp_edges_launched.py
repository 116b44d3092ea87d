"""The step of systems whose chains cross the edges of warps and tiles by every
route: in one kernel, by launches with the pair kernel, and by launches whose
stages walk the lists.  The systems, the oracle's step and the tolerance (1e-13)
are those of ``test_gpu_warp_edges``, which small systems meet in one kernel
whatever their pair mode.

SRK4 and mixed precision against the one-kernel steps, which sum in the same
order: equal bits, with chain lengths that do not divide 32."""
import copy

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests.golden_io import min_image  # noqa: E402
from tests.test_gpu_warp_edges import _spec  # noqa: E402


@pytest.mark.parametrize("dim,cutoff", [(2, 1.0), (2, W.LJ_CUTOFF), (3, 1.0), (3, W.LJ_CUTOFF)])
@pytest.mark.parametrize("n,length", [(2, 2), (33, 33), (63, 5), (64, 31), (65, 16), (129, 32), (130, 7), (385, 40)])
def test_a_step_by_every_route(dim, cutoff, n, length):
    spec = _spec(dim, n, length, cutoff)
    p = spec.params
    ng = max(1, int(p.L / (2.0 * max(1.0, p.wca_params[3]))))
    o = O.OracleSystem(spec.pos, spec.tangent, spec.chain_id, spec.rest_lengths, p.L, p.spring_params, p.wca_params,
                       p.active_params, p.D, p.Dr, p.radius, p.n_nearby, ng, nbor_depth=256)
    o.build_lists(grid_window=max(1, int(np.ceil(p.wca_params[3] / (p.L / ng)))))
    o.run(1, dt=1e-4, dtmax=p.dtmax, max_dist_per_step=p.max_dist_per_step, noise_mode=O.NOISE_PHILOX, seed=p.seed)
    for ctas in (0, -1):
        for mode, block in ((0, 128), (0, 64), (1, 128), (1, 64)):
            b = Batch([spec], precision="fp64", pair_mode=mode, block_beads=block, ctas_per_sm=ctas, list_depth=128)
            b.begin(1, dt=1e-4)
            before = b.engine.launches()
            b.run(1)
            assert b.engine.launches() - before == (2 if ctas == 0 else 2 + 10 * (10 if mode == 1 else 12))
            st = b.statuses()[0]
            assert st["steps_done"] == 1 and st["flags"] == 0
            err = np.max(np.abs(min_image(b.states[0].pos.cpu().numpy() - o.pos, p.L)))
            assert err < 1e-13, (ctas, mode, block, err)
            b.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("order,mode", [(2, 0), (2, 1), (4, 0)])
@pytest.mark.parametrize("n_chains,clen", [(70, 7), (41, 13), (9, 45), (13, 31)])
def test_launches_as_in_one_kernel(precision, dim, order, mode, n_chains, clen):
    spec = W.make_system("s", dim, n_chains, clen, 40.0 if dim == 2 else 18.0, seed=clen, T=0.1,
                         v_tan_angle=0.2 if dim == 2 else 0.0)
    out = []
    for ctas in (0, -1):
        b = Batch([copy.deepcopy(spec)], precision=precision, srk_order=order, pair_mode=mode, ctas_per_sm=ctas)
        b.set_adaptive(True)
        b.begin(20, dt=1e-4)
        b.run(20)
        out.append([b.big[k].cpu().numpy() for k in ("pos", "pos1", "forces", "tangent")])
        b.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
