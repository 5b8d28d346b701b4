"""The face flux by two lanes on both sides of the mesh size at which one
thread per face takes over (85248 faces), and where the last warp of a
direction is partly empty: one step equals the oracle's bit for bit."""
import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import Solver, root_keys

pytestmark = pytest.mark.gpu


# interior base x base: 2 base (base + 1) faces
@pytest.mark.parametrize("base", [7, 13, 64, 205, 206, 207])
def test_step_equals_the_oracle(oracle_mod, base):
    cfg = P.riemann4(base=base, lvl_amr=0)
    keys = root_keys(cfg.m, cfg.n)
    rng = np.random.default_rng(base)
    prim = rng.uniform([0.5, -1.0, -1.0, 0.5], [1.5, 1.0, 1.0, 1.5], size=(len(keys), 4))
    prim[len(keys) // 2:len(keys) // 2 + 5, 1] = 1e-300   # refused by the branch-free division: one lane of a pair or both
    o = oracle_mod.Oracle(cfg, initial=False)
    g = Solver(cfg)
    o.set_leaves(keys, prim)
    g.upload(keys, prim)
    for s in (o, g):
        s.set_scalars(3.0, 3.0, 1e-4, 0.0, 0)
    o.time_advance_rk()
    g.time_advance_rk(1e-4)
    assert np.array_equal(g.leaves()[1], o.leaves()[1])
    g.close()
