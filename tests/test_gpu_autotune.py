"""The autotuner times each launch shape of the face kernel once: the variant
numbers past the six shapes repeat their shape's time, and the number that it
keeps is a shape's own."""
import numpy as np
import pytest

from fdm_cell_based_amr_cartesian_b200 import params as P
from fdm_cell_based_amr_cartesian_b200.solver import FACE_VARIANTS, Solver

pytestmark = pytest.mark.gpu
SHAPES = 6


@pytest.mark.parametrize("flux", [0, 1])
def test_each_shape_is_timed_once(flux):
    cfg = P.riemann4(base=64, lvl_amr=0)
    cfg.params.flux_variant = flux
    g = Solver(cfg)
    g.creat_mesh_and_initial()
    best, ms = g.autotune(reps=3)
    assert len(ms) == FACE_VARIANTS and (ms > 0).all()
    assert np.array_equal(ms, ms[np.arange(FACE_VARIANTS) % SHAPES])
    assert best < SHAPES and ms[best] == ms.min()
    for v in range(FACE_VARIANTS):      # every old number is taken still
        g.set_variant(v)
    g.close()
