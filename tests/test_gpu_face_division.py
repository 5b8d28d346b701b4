"""The face flux's branch-free division where it refuses operands: states
whose densities, pressures or velocities leave its exact ranges are computed
again with the compiler's division, and every face equals the oracle's bit
for bit either way."""
import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import Solver, root_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,refused", [
    ("ordinary", "none"),
    ("density and pressure times 2^-120", "all"),      # below the range of the mean density
    ("pressure times 2^120", "all"),                   # sound speed above the range
    ("one velocity of 1e-300", "some"),                # numerators whose remainders would underflow
    ("a velocity of zero", "none"),
    ("constant state", "none"),                        # smoothness indicators of rounding noise
])
def test_faces_equal_the_oracle(oracle_mod, case, refused):
    cfg = P.riemann4(base=13, lvl_amr=0)   # 19 x 19 cells, 13 x 14 and 14 x 13 faces: partial blocks
    rng = np.random.default_rng(7)
    keys = root_keys(cfg.m, cfg.n)
    prim = rng.uniform([0.5, -1.0, -1.0, 0.5], [1.5, 1.0, 1.0, 1.5], size=(len(keys), 4))
    if case.startswith("density"):
        prim[:, [0, 3]] *= 2.0 ** -120
    elif case.startswith("pressure"):
        prim[:, 3] *= 2.0 ** 120
    elif case.startswith("one velocity"):
        prim[:, 2] = 0.0
        prim[len(keys) // 2 - 40:len(keys) // 2, 2] = 1e-300
    elif case.startswith("a velocity"):
        prim[:, 1] = 0.0
    elif case.startswith("constant"):
        prim[:] = prim[0]
    dt = 1e-3 if not case.startswith("pressure") else 1e-21
    o = oracle_mod.Oracle(cfg, initial=False)
    o.set_leaves(keys, prim)
    o.set_scalars(3.0, 3.0, dt, 0.0, 0)
    g = Solver(cfg)
    g.upload(keys, prim)
    g.set_scalars(3.0, 3.0, dt, 0.0, 0)
    nx, ny = g.nr_fallbacks()
    faces = 14 * 13
    assert {"none": nx + ny == 0, "all": nx + ny == 2 * faces, "some": 0 < nx + ny < 2 * faces}[refused], (nx, ny)
    o.time_advance_rk()
    g.time_advance_rk(dt)
    _, po, _ = o.leaves()
    _, pg = g.leaves()
    assert np.all(np.isfinite(po))
    assert np.array_equal(pg, po)
    g.close()
