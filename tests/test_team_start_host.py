"""The one-kernel steps write into the shared memory of the other CTAs of a
cluster, which is defined only once every CTA of it has started: the kernel
meets at the cluster's barrier before anything else that may write there."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gliding_collective_rotation_b200",
                    "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as fh:
        return re.sub(r"//[^\n]*", "", fh.read())


def _body(src, head):
    """The braces that follow ``head``."""
    at = src.index("{", src.index(head))
    depth = 0
    for k in range(at, len(src)):
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        if depth == 0:
            return src[at:k + 1]
    raise AssertionError(head)


def test_clusters_meet_before_the_first_remote_store():
    src = _source("gcr_phases.cuh")
    # Team::sync is the only writer of another CTA's shared memory ...
    assert src.count("store_cluster(") == 1 + _body(src, "struct Team {").count("store_cluster(")
    # ... k_steps the only kernel with a team, and its first barrier comes first
    assert len(re.findall(r"\bTeam team\{", src)) == 1
    body = _body(src, "k_steps(const")
    meet, sync = body.find("cluster_sync();"), body.index("team.sync(")
    assert 0 <= meet < sync
    assert "return" not in body[:meet] and "team_" not in body[:meet] and "{" not in body[body.index("Span"):meet]
