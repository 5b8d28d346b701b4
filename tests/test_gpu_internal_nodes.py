"""Internal nodes and their interpA means after an upload, against a numpy
restatement bit for bit: the ancestors named by the leaves' trailing zero
digits, for sorted and shuffled leaf sets, a bare background grid and deep
random trees."""
import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import Solver, root_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("base,lvl,prob,shuffled", [
    (3, 0, 0.0, False),      # no internal node
    (3, 5, 0.5, True),
    (19, 3, 0.3, False),
    (19, 3, 0.3, True),
    (64, 4, 0.25, False),
])
def test_internal_nodes_after_upload(base, lvl, prob, shuffled):
    cfg = P.riemann4(base, max(lvl, 1))
    rng = np.random.default_rng(base + lvl)
    keys, inner = root_keys(cfg.m, cfg.n), np.zeros(0, np.uint64)
    son = lambda k, q, level: (k | (np.uint64(q) << np.uint64(4 + 2 * (14 - level)))) + np.uint64(1)
    for level in range(lvl):
        hit = ((keys & np.uint64(15)) == level) & (rng.random(len(keys)) < prob)
        inner = np.concatenate([inner, keys[hit]])
        keys = np.sort(np.concatenate([keys[~hit]] + [son(keys[hit], q, level) for q in range(4)]))
    inner = np.sort(inner)
    prim = rng.uniform([0.5, -1.0, -1.0, 0.5], [1.5, 1.0, 1.0, 1.5], size=(len(keys), 4))
    value = dict(zip(keys.tolist(), prim))
    for k in inner[np.argsort(inner & np.uint64(15), kind="stable")[::-1]]:
        level = int(k & np.uint64(15))
        c = [value[int(son(k, q, level))] for q in range(4)]
        value[int(k)] = 0.25 * (c[0] + c[1] + c[3] + c[2])
    order = rng.permutation(len(keys)) if shuffled else np.arange(len(keys))
    g = Solver(cfg)
    g.upload(keys[order], prim[order])
    ik, iv = g.internal_nodes()
    assert np.array_equal(ik, inner)
    if len(inner):
        assert np.array_equal(iv, np.stack([value[int(k)] for k in inner]))
    kg, pg = g.leaves()
    assert np.array_equal(kg, keys) and np.array_equal(pg, prim)
    g.close()
