"""gridmodify4 with too little room for its new nodes: the pass is taken again
with more, and ends on the oracle's leaf set, values and counts.  A room of 4
holds the sons of one refinement; the usual one (0) and one of 64 nodes stand
beside it."""
import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import Solver
from test_gpu_gridmodify4 import _random_tree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [4, 64, 0])
def test_a_pass_that_fills_its_pool_is_taken_again(oracle_mod, nodes):
    cfg = P.riemann4(17, 4)
    cfg.params.refine_goal_rot = cfg.params.refine_goal_div = 1.0
    cfg.params.coarse_goal_rot = cfg.params.coarse_goal_div = 0.05
    rng = np.random.default_rng(174)
    keys = _random_tree(cfg, 4, 0.2, rng)
    o = oracle_mod.Oracle(cfg, initial=False)
    g = Solver(cfg)
    assert g.L.fdm_debug_gm4_pool(g.h, nodes) == 0
    for _ in range(2):
        prim = rng.uniform([0.5, -1.0, -1.0, 0.5], [1.5, 1.0, 1.0, 1.5], size=(len(keys), 4))
        for s in (o, g):
            (s.set_leaves if s is o else s.upload)(keys, prim)
            s.set_scalars(0.0, 0.0, 1e-4, 0.0, 0)
            s.amr()
        g.body_boundary(1)
        kg, pg = g.leaves()
        keys, po, _ = o.leaves()
        assert np.array_equal(kg, keys)
        assert np.array_equal(pg, po)
        assert g.counters()["n_gm4_nonleaf"] == o.counters()["gm4_nonleaf"]
    assert g.counters()["n_gm4_refines"] > 16      # more than either small room holds in one pass
    g.close()
