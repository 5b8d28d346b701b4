"""The no-allocation step equals the handle's time_advance_rk on the same
uniform periodic leaf set bit for bit, also where the branch-free division
refuses operands (scaled density and pressure)."""
import ctypes

import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import Solver, load_library, root_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -120, 2.0 ** 120])
def test_bits_of_the_handle_path(scale):
    import torch

    cfg = P.vortex(lvl_amr=0)             # 32 x 32 interior, periodic
    p = cfg.params
    keys = root_keys(cfg.m, cfg.n)
    prim = np.random.default_rng(9).uniform([0.5, -1.0, -1.0, 0.5], [1.5, 1.0, 1.0, 1.5], size=(len(keys), 4))
    prim[:, [0, 3]] *= scale
    g = Solver(cfg)
    g.upload(keys, prim)
    g.body_boundary(1)                    # periodic ghosts
    _, u0 = g.leaves()
    g.set_scalars(3.0, 3.0, 1e-3, 0.0, 0)
    cur = torch.tensor(u0, dtype=torch.float64, device="cuda")
    out = torch.empty_like(cur)
    rc = load_library().fdm_time_advance_rk_uniform_static(
        cur.data_ptr(), out.data_ptr(), cfg.m - 6, cfg.n - 6, p.h, p.x_factor, p.gama, 3.0, 3.0, 1e-3,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    g.time_advance_rk(1e-3)
    ref = g.leaves()[1]
    got = out.cpu().numpy()
    assert np.isfinite(ref).all()
    assert np.array_equal(got, ref), np.argwhere(got != ref)[:4]
    g.close()
