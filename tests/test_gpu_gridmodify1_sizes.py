"""gridmodify1 on both sides of the node-set size at which it changes from one
cluster launch to a launch per sweep (32768 nodes): two regrids equal the
oracle's."""
import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import Solver

pytestmark = pytest.mark.gpu


# (base + 6)^2 cells with their ghosts, before any refinement
@pytest.mark.parametrize("base,cluster", [(40, True), (160, True), (180, False)])   # 2116, 27556 and 34596 nodes
def test_regrids_equal_the_oracle(oracle_mod, base, cluster):
    cfg = P.riemann4(base=base, lvl_amr=2)
    o = oracle_mod.Oracle(cfg)
    g = Solver(cfg)
    g.creat_mesh_and_initial()
    for k in range(2):
        o.solute(2)
        assert g.solute(2) == 2
        o.amr()
        g.amr()
        g.body_boundary(1)
        assert ((base + 6) ** 2 <= 32768) == cluster
        (kg, pg), (ko, po, _) = g.leaves(), o.leaves()
        assert np.array_equal(kg, ko), (len(kg), len(ko))
        assert np.array_equal(pg, po)
    g.close()
