"""gridmodify4 by its fixpoint of refinement times against the oracle's
recursive traversal, on trees far rougher than a flow makes: cells refined at
random to any depth, so that cascades, leaves made ahead of and behind the
traversal, grid edges and dozens of refinements of nodes that have sons meet
in one pass.  Bit-exact: the leaf set, the values and the count of such
refinements."""
import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import Solver, root_keys

pytestmark = pytest.mark.gpu


def _random_tree(cfg, lvl, prob, rng):
    keys = root_keys(cfg.m, cfg.n)
    for level in range(lvl):
        hit = ((keys & np.uint64(15)) == level) & (rng.random(len(keys)) < prob)
        sons = [(keys[hit] | (np.uint64(q) << np.uint64(4 + 2 * (14 - level)))) + np.uint64(1) for q in range(4)]
        keys = np.sort(np.concatenate([keys[~hit]] + sons))
    return keys


@pytest.mark.parametrize("problem,base,lvl,prob", [
    ("riemann4", 3, 5, 0.4),       # 9 x 9 background cells, deep
    ("riemann4", 17, 4, 0.2),
    ("vortex", 16, 3, 0.4),        # periodic
    ("double_mach", 7, 4, 0.4),    # 34 x 13
    ("riemann4", 61, 4, 0.2),      # more looks than the cluster has threads
])
def test_rough_regrids_match_the_traversal(oracle_mod, problem, base, lvl, prob):
    cfg = {"riemann4": P.riemann4, "vortex": P.vortex, "double_mach": P.double_mach}[problem](base, lvl)
    cfg.params.refine_goal_rot = cfg.params.refine_goal_div = 1.0
    cfg.params.coarse_goal_rot = cfg.params.coarse_goal_div = 0.05
    rng = np.random.default_rng(base * 10 + lvl)
    keys = _random_tree(cfg, lvl, prob, rng)
    o = oracle_mod.Oracle(cfg, initial=False)
    g = Solver(cfg)
    for k in range(3):
        prim = rng.uniform([0.5, -1.0, -1.0, 0.5], [1.5, 1.0, 1.0, 1.5], size=(len(keys), 4))
        o.set_leaves(keys, prim)
        o.set_scalars(0.0, 0.0, 1e-4, 0.0, 0)
        g.upload(keys, prim)
        g.set_scalars(0.0, 0.0, 1e-4, 0.0, 0)
        o.amr()
        g.amr()
        g.body_boundary(1)
        kg, pg = g.leaves()
        keys, po, _ = o.leaves()
        assert np.array_equal(kg, keys), f"round {k}: leaf sets differ ({len(kg)} vs {len(keys)})"
        assert np.array_equal(pg, po), f"round {k}: values differ"
        assert g.counters()["n_gm4_nonleaf"] == o.counters()["gm4_nonleaf"], f"round {k}"
    assert g.counters()["n_gm4_refines"] > 0
    g.close()
