"""A new descriptor for a resident system: the same one again changes nothing,
one that leaves the list radius, skin, box and exclusions alone keeps the
lists, any other rebuilds them -- and every one steps on bit for bit as a fresh
context given the same state and parameters does."""
import copy

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from gliding_collective_rotation_b200 import workloads as W  # noqa: E402
from gliding_collective_rotation_b200.batch import Batch  # noqa: E402


def _change(p, what):
    if what == "none":
        pass
    elif what == "noise":
        p.D, p.dtmax, p.rk_cheat = 0.02, 5e-4, 0.9
    elif what == "springs":
        p.spring_params = p.spring_params * np.array([1.1, 0.9, 1.0, 1.0, 1.0, 1.0])
    elif what == "cutoff":
        p.wca_params = p.wca_params * np.array([1.0, 1.0, 1.0, 1.1])
    elif what == "skin":
        p.skin = 0.5
    elif what == "exclusions":
        p.n_nearby = 2


@pytest.mark.parametrize("ctas", [0, -1])
@pytest.mark.parametrize("what,rebuilds", [("none", False), ("noise", False), ("springs", False), ("cutoff", True),
                                           ("skin", True), ("exclusions", True)])
def test_new_descriptor(what, rebuilds, ctas):
    spec = W.make_system("s", 2, 150, 8, 50.0, 4)
    b = Batch([copy.deepcopy(spec)], precision="fp64", ctas_per_sm=ctas)
    b.relax(max_steps=600, adaptive_after=True)
    st = b.states[0]
    before = b.statuses()[0]
    kept = [b.big[k].clone() for k in ("pos", "tangent")]
    b.begin(1, dt=before["dt"])
    b.run(1)
    unchanged = b.statuses()[0]["list_builds"] - before["list_builds"]
    if unchanged:
        pytest.skip("the step leaves a skin by itself")
    for k, v in zip(("pos", "tangent"), kept):
        b.big[k].copy_(v)
    before = b.statuses()[0]
    _change(st.params, what)
    b.engine.update_params(st)
    later = copy.deepcopy(spec)
    later.params = copy.deepcopy(st.params)
    later.params.step = before["step"]
    later.pos, later.tangent = st.pos.cpu().numpy(), st.tangent.cpu().numpy()
    fresh = Batch([later], precision="fp64", ctas_per_sm=ctas)
    for x in (b, fresh):
        x.begin(1, dt=before["dt"])
        x.run(1)
    one = b.statuses()[0]["list_builds"] - before["list_builds"]
    for x in (b, fresh):
        x.begin(9)
        x.run(9)
    for k in ("pos", "pos1", "tangent", "forces"):
        assert torch.equal(b.big[k], fresh.big[k]), k
    assert b.statuses()[0]["flags"] == 0 and b.statuses()[0]["steps_done"] == 9
    if rebuilds:
        assert one >= 1
    else:
        # a build in this one step only if a bead left its skin in it
        assert one == unchanged
    b.close()
    fresh.close()
