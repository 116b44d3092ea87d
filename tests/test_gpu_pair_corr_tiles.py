"""Pair correlations on the GPU against the CPU restatement at the edges of the
kernel's tiles (64 chains, four a CTA, in 16 to 1 slices) and of its bins.

Single-bead chains: a chain's centre is its bead.  On the lattice every
distance along an axis lies exactly on a bin's edge, where the FP32 quotient
cannot decide.  Counts are whole, so g(r) agrees to the rounding of its
normalisation (1e-12); the Cvv and Cnn sums hold 2^-32 a pair, so their means
agree within 2^-32 and rounding (1e-9).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import observables as OBS  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402
from gliding_collective_rotation_b200.engine import SystemParams, wca_params  # noqa: E402
from gliding_collective_rotation_b200.workloads import SystemSpec  # noqa: E402
from oracle import observables as OB  # noqa: E402


@pytest.mark.parametrize("n", [2, 63, 64, 65, 128, 129, 257, 700, 1000, 1400, 1500, 2300])
@pytest.mark.parametrize("lattice,binsize", [(False, 0.25), (True, 0.25), (False, 0.1), (True, 0.1)])
def test_pair_correlation_at_tile_and_bin_edges(n, lattice, binsize):
    rs = np.random.default_rng([n, lattice])
    L = 16.0
    pos = rs.integers(0, 64, size=(n, 2)) * 0.25 if lattice else rs.uniform(0, L, size=(n, 2))
    a = rs.uniform(0, 2 * np.pi, n)
    prm = SystemParams(L=L, spring_params=np.zeros(6), wca_params=wca_params(0.1, 1.0, 0.0, 1.0),
                       active_params=np.zeros(3), D=0.0, Dr=0.0, radius=0.1, n_nearby=0, calc_springs=False)
    spec = SystemSpec("points", 2, pos, np.stack([np.cos(a), np.sin(a)], axis=1), np.arange(n), np.full(n, 0.5), prm,
                      1e-3, 0.0125)
    b = Batch([spec], precision="fp64")
    eng, slot = b.engine, b.states[0].slot
    com, phi = OBS.chain_frames(eng, slot)
    assert np.array_equal(com, pos)
    for kind, k, tol in (("g_of_r", 0, 1e-12), ("Cvv", 1, 1e-9), ("Cnn", 2, 1e-9)):
        got = OBS.pair_correlation(eng, slot, kind, binsize)
        want = OB.correlation(com, L, k, binsize, phi[:, 0], phi[:, 1])
        assert got.shape == want.shape
        assert np.allclose(got, want, rtol=tol, atol=tol, equal_nan=True), kind
    b.close()
