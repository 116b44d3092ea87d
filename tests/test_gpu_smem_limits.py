"""Contexts whose kernels take different amounts of dynamic shared memory, alive
at once: the limit of a kernel is every context's, so none may lower another's.
Each steps on after the others have run, as it does alone."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402

KW = {"lists": [dict(list_depth=96), dict(list_depth=32)],
      "blocks": [dict(block_beads=512, list_depth=96), dict(block_beads=64)],
      "cells": [dict(block_beads=512, pair_mode=2), dict(block_beads=128, pair_mode=2)],
      "wide": [dict(block_beads=512), dict(block_beads=128)]}


def _step(b):
    b.begin(10)
    b.run(10)
    torch.cuda.synchronize()
    assert all(s["flags"] == 0 and s["steps_done"] == 10 for s in b.statuses())


def _batch(dim, kw):
    spec = W.make_system("s", dim, 150, 7, 40.0 if dim == 2 else 20.0, seed=4)
    b = Batch([spec], precision="fp64", **kw)
    b.set_adaptive(True)
    return b


@pytest.mark.parametrize("first", [0, 1])
@pytest.mark.parametrize("dim,what", [(2, "lists"), (3, "lists"), (2, "blocks"), (3, "blocks"), (2, "cells"),
                                      (3, "cells"), (3, "wide")])
def test_contexts_step_in_turn(dim, what, first):
    kws = KW[what] if first == 0 else KW[what][::-1]
    alone = []
    for kw in kws:
        b = _batch(dim, kw)
        _step(b)
        _step(b)
        alone.append(b.states[0].pos.cpu().numpy())
        b.close()
    bs = [_batch(dim, kw) for kw in kws]
    for _ in range(2):
        for b in bs:
            _step(b)
    for b, want in zip(bs, alone):
        np.testing.assert_array_equal(b.states[0].pos.cpu().numpy(), want)
        b.close()
