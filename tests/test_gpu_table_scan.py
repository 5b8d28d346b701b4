"""The prefix sums of the table build where their tiles and their method
change: 8 flags per interior leaf, in tiles of 8192 by one block or a cluster
of up to eight, up to 524288 flags.  A mesh with scattered cells refined once;
one step equals the oracle's bit for bit."""
import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import Solver, root_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("base,refined", [
    (12, 3),       # 153 interior leaves
    (29, 61),      # 1024: one full tile
    (29, 62),      # 1027
    (80, 604),     # 8212: just above eight tiles
    (200, 8512),   # 65536: the largest by a cluster
    (200, 8513),   # 65539
])
def test_step_equals_the_oracle(oracle_mod, base, refined):
    cfg = P.riemann4(base=base, lvl_amr=1)
    rng = np.random.default_rng(base + refined)
    roots = root_keys(cfg.m, cfg.n)
    m = cfg.m
    rows, cols = np.divmod((roots >> np.uint64(34)).astype(np.int64), m)
    inner = (rows >= 6) & (rows < cfg.n - 6) & (cols >= 6) & (cols < m - 6)
    pick = rng.choice(np.flatnonzero(inner), size=refined, replace=False)
    keep = np.ones(len(roots), bool)
    keep[pick] = False
    sons = (roots[pick][:, None] | (np.arange(4, dtype=np.uint64) << np.uint64(32))[None, :] | np.uint64(1)).ravel()
    keys = np.sort(np.concatenate([roots[keep], sons]))
    prim = rng.uniform([0.5, -1.0, -1.0, 0.5], [1.5, 1.0, 1.0, 1.5], size=(len(keys), 4))
    o = oracle_mod.Oracle(cfg, initial=False)
    g = Solver(cfg)
    o.set_leaves(keys, prim)
    g.upload(keys, prim)
    assert g.counters()["n_interior"] == base * base + 3 * refined
    for s in (o, g):
        s.set_scalars(3.0, 3.0, 1e-5, 0.0, 0)
    o.time_advance_rk()
    g.time_advance_rk(1e-5)
    assert np.array_equal(g.leaves()[1], o.leaves()[1])
    g.close()
