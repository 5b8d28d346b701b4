"""Instructions of the aligned form (cluster barriers, matrix ones) want all lanes of a warp
to execute them together; after lane-dependent code nothing promises that but
a __syncwarp().  Read from the kernels' source, since a violation is undefined
behaviour that a run need not show."""
import glob
import os
import re

import pytest

from fdm_cell_based_amr_cartesian_b200 import build as B


def _statements(path):
    txt = re.sub(r"//[^\n]*", "", open(path).read())
    return [s.strip() for s in re.split(r"(?<=[;{}])\s*\n", txt) if s.strip()]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(B.CSRC, "*.cu*"))), ids=os.path.basename)
def test_cluster_barriers_follow_a_warp_barrier(path):
    st = _statements(path)
    for before, s in zip(st, st[1:]):
        if "barrier.cluster" in s and ".aligned" in s:
            assert before.endswith("__syncwarp();"), (os.path.basename(path), s)


def test_gate_fragments_are_read_before_a_warp_barrier():
    """w3 is read by the lanes with g == 0 only, and the next instruction may be
    a matrix one (k_mlp_eval, the transposes of k_mlp_grad)."""
    txt = open(os.path.join(B.CSRC, "gate_items.cuh")).read()
    body = re.search(r"explicit GateFrag\(const GateWeights &W\) \{\n(.*?)\n    \}\n", txt, re.S).group(1)
    last = [ln.strip() for ln in body.splitlines() if ln.strip()][-1]
    assert "g == 0" in body and last.startswith("__syncwarp();"), last
