"""gridmodify1 where its path and its loops change, with the side read from the
counters around each regrid: a cluster of 16384 threads takes node sets of up
to 32768 (so most threads a second node here), a launch per sweep the larger
ones.  Leaf sets and values equal the oracle's bit for bit."""
import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import Solver

pytestmark = pytest.mark.gpu
CLUSTER_THREADS, CLUSTER_MAX = 16384, 32768


def _nodes(g):
    c = g.counters()
    return c["n_leaves"] + c["n_internal"]


@pytest.mark.parametrize("base,lo,hi", [
    (120, CLUSTER_THREADS, CLUSTER_MAX),
    (130, CLUSTER_THREADS, CLUSTER_MAX),   # ends just below the limit
    (180, CLUSTER_MAX, 1 << 31),
])
def test_regrids_equal_the_oracle(oracle_mod, base, lo, hi):
    cfg = P.riemann4(base=base, lvl_amr=2)
    o = oracle_mod.Oracle(cfg)
    g = Solver(cfg)
    g.creat_mesh_and_initial()
    for _ in range(2):
        o.solute(2)
        assert g.solute(2) == 2
        assert lo < _nodes(g) <= hi
        o.amr()
        g.amr()
        assert lo < _nodes(g) <= hi
        g.body_boundary(1)
        (kg, pg), (ko, po, _) = g.leaves(), o.leaves()
        assert np.array_equal(kg, ko), (len(kg), len(ko))
        assert np.array_equal(pg, po)
    assert g.counters()["n_gm1_iterations"] > 0
    g.close()
