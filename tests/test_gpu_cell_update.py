"""The cell update on both sides of the mesh size at which its kernel changes
(592 blocks of 256 leaves), and the no-allocation step where the branch-free
division refuses operands: equal to the oracle bit for bit."""
import ctypes

import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import Solver, load_library, root_keys

pytestmark = pytest.mark.gpu


def _state(n, scale, seed=5):
    rng = np.random.default_rng(seed)
    prim = rng.uniform([0.5, -1.0, -1.0, 0.5], [1.5, 1.0, 1.0, 1.5], size=(n, 4))
    prim[:, [0, 3]] *= scale
    return prim


@pytest.mark.parametrize("base", [389, 390])   # 151321 leaves: 592 blocks; 152100: 595
def test_step_at_the_kernel_change(oracle_mod, base):
    cfg = P.riemann4(base=base, lvl_amr=0)
    keys = root_keys(cfg.m, cfg.n)
    prim = _state(len(keys), 1.0)
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


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -120, 2.0 ** 120])   # of density and pressure
def test_uniform_step(oracle_mod, scale):
    import torch

    cfg = P.vortex(lvl_amr=0)             # 32 x 32 interior, periodic
    p = cfg.params
    keys = root_keys(cfg.m, cfg.n)
    prim = _state(len(keys), scale)
    o = oracle_mod.Oracle(cfg, initial=False)
    g = Solver(cfg)
    o.set_leaves(keys, prim)
    g.upload(keys, prim)
    g.body_boundary(1)                    # periodic ghosts
    _, u0 = g.leaves()
    o.set_leaves(keys, u0)
    o.set_scalars(3.0, 3.0, 1e-3, 0.0, 0)
    cur = torch.tensor(u0, dtype=torch.float64, device="cuda")
    out = torch.empty_like(cur)
    rc = load_library().fdm_time_advance_rk_uniform_static(
        cur.data_ptr(), out.data_ptr(), cfg.m - 6, cfg.n - 6, p.h, p.x_factor, p.gama, 3.0, 3.0, 1e-3,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    o.time_advance_rk()
    ref = o.leaves()[1]
    assert np.max(np.abs(out.cpu().numpy() - ref) / np.maximum(np.abs(ref), 1e-14 * min(scale, 1.0))) <= 1e-12
    g.close()
