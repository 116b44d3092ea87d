"""Small batches step in one kernel whose CTAs meet at barriers; one CTA per
tile (``ctas_per_sm=-1``) steps the same batch launch by launch.  Both run the
same phases in the same order, so states, statuses and series are equal bit
for bit: for one tile, a full cluster (16 tiles), one tile more (clusters that
meet in global memory), a ragged last cluster, every SRK order and option, calls
cut by steps or by time, and lists that overflow and are regrown."""
import copy

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402


def _state(b):
    torch.cuda.synchronize()
    out = [b.big[k].cpu().numpy() for k in sorted(b.big) if k not in ("chain_id", "rest")]
    return out + [u.cpu().numpy() for u in b.unwrapped()] + [np.array([list(s.values()) for s in b.statuses()])]


def _both(specs, program, precision="mixed", couple=(), motors=(), **kw):
    got = []
    for ctas in (-1, 0):
        b = Batch([copy.deepcopy(s) for s in specs], precision=precision, ctas_per_sm=ctas, **kw)
        for g in couple:
            b.couple(*g)
        for m in motors:
            b.set_motors(*m)
        b.set_adaptive(True)
        extra = program(b)
        got.append(_state(b) + ([] if extra is None else [extra]))
        b.close()
    for x, y in zip(*got):
        assert x.shape == y.shape and np.array_equal(x, y, equal_nan=True)


def _run(b):
    b.begin(45, dt=1e-4)
    b.run(20)
    b.run(25)


def _system(dim, n_chains, clen=8, seed=3, **kw):
    L = 60.0 if dim == 2 else 24.0
    return W.make_system("s", dim, n_chains, clen, L, seed, **kw)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("dim,n_chains", [(2, 1), (2, 9), (2, 256), (2, 257), (2, 1000), (3, 16), (3, 300)])
def test_sizes(dim, n_chains, precision):
    _both([_system(dim, n_chains, v_tan_angle=0.2 if dim == 2 else 0.0)], _run, precision)


def test_several_systems_with_series_and_lj():
    specs = [_system(2, 40, seed=1), _system(2, 333, clen=5, seed=2, eps=0.5, cutoff=W.LJ_CUTOFF),
             _system(2, 111, clen=13, seed=4)]

    def program(b):
        b.begin(60, dt=1e-4, series_every=7)
        b.run(60)
        return np.concatenate(b.series())

    _both(specs, program, list_depth=128)


def test_rotational_diffusion_and_rigid_rods():
    free = _system(3, 100, seed=5, tangent_locked=False, Dr=0.1)
    rods = _system(2, 120, seed=6)
    rods.params.rigid_rod = 0.5
    _both([free], _run)
    _both([rods], _run, "fp64")


@pytest.mark.parametrize("dim", [2, 3])
def test_srk4(dim):
    s = _system(dim, 130, seed=7)
    s.params.rigid_rod = 0.3 if dim == 2 else 0.0
    _both([s, _system(dim, 20, seed=8)], _run, "fp64", srk_order=4)


def test_coupled_populations_and_motors():
    specs, groups = W.populations(1, seed=2)
    _both(specs, _run, couple=groups)
    fixed = [(groups[0][0], [False, True], groups[0][2])]
    _both(specs, _run, "fp64", couple=fixed)
    specs, groups, mots = W.motors(2, seed=3, n_chains=60, L=40.0)
    _both(specs, _run, couple=groups, motors=mots, list_depth=128)


def test_calls_cut_by_time_and_overflows():
    def timed(b):
        b.begin(-1, dt=1e-4, max_dt_usable=2e-3)
        b.run(1 << 62, sync_every=1)

    _both([_system(2, 300, seed=9), _system(2, 30, seed=10)], timed, "fp64")

    def checked(b):
        sts = b.run_checked(60)
        assert all(s["steps_done"] == 60 for s in sts)

    _both([_system(2, 400, seed=11, eps=0.5, cutoff=W.LJ_CUTOFF)], checked, "fp64", list_depth=4)
