"""The last block of a grid team to arrive adds up the others' partial sums with a
whole warp, while one lane has counted the block in: the lanes may read only
after a barrier of the warp that follows that lane's acquire (a shuffle orders
no memory).  Read from the source."""
import os
import re

from dare_b200.build import CSRC


def test_lanes_read_after_the_acquire():
    with open(os.path.join(CSRC, "dare_team.cuh")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    team = text[text.index("struct GridTeam"):text.index("struct ClusterTeam")]
    acquire = team.index("atom.acq_rel.gpu")
    read = team.index("ld.relaxed.gpu.global.f64", acquire)
    assert "__syncwarp()" in team[acquire:read]
