"""Kernels whose blocks form a cluster wait for one another before the first
access to another block's shared memory: the blocks are placed together but
need not have started together.  Read from the sources, since a run that
happens to pass does not show it."""
import glob
import os
import re

import pytest

from dare_b200.build import CSRC

TEAM = os.path.join(CSRC, "dare_team.cuh")


def _source(path):
    with open(path) as f:
        text = re.sub(r"/\*.*?\*/", "", f.read(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _block(text, at):
    """The braces' contents that open at or after `at`."""
    i = text.index("{", at)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i + 1:j]
        j += 1


def _kernels():
    """(file, body) of every kernel that makes a cluster team."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = _source(path)
        for m in re.finditer(r"__global__", text):
            body = _block(text, text.index(")", text.index("k_", m.start())))
            if "ClusterTeam::here" in body:
                out.append((os.path.basename(path), body))
    return out


def test_start_is_a_barrier_of_the_cluster():
    team = _source(TEAM)
    cluster = _block(team, team.index("struct ClusterTeam"))
    assert re.search(r"\bbarrier\(\)", _block(cluster, cluster.index("void start()")))
    barrier = _block(cluster, cluster.index("void barrier()"))
    assert "barrier.cluster.arrive.release" in barrier and "barrier.cluster.wait.acquire" in barrier


def test_every_cluster_kernel_is_found():
    assert [f for f, _ in _kernels()] == ["dare_batched.cu", "dare_resident.cu"]


@pytest.mark.parametrize("file,body", _kernels(), ids=lambda v: v if v.endswith(".cu") else "")
def test_kernels_start_their_team_first(file, body):
    start = body.index("team.start()")
    for use in (r"ClusterTeam::remote", r"team\.(?:template )?sum", r"shared::cluster", r"team_iterations"):
        for m in re.finditer(use, body):
            assert m.start() > start, (file, use)
