"""Lines long enough that the untuned solver takes 8 problems a block: bit for
bit the same as with 16, whose blocks hold the same segments."""
import math

import numpy as np
import pytest

from ekcases import sheared_case, small_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,ny2,nz2,nprob", [
    (small_case, 289, 33, 201), (small_case, 321, 33, 147), (small_case, 385, 33, 200), (small_case, 33, 385, 200),
    (sheared_case, 33, 321, 200), (small_case, 385, 33, 5)])
def test_eight_problems_a_block(case, ny2, nz2, nprob):
    p, xp, yp, _ = case(16, ny2, nz2)
    p.mg_stop, p.mg_tol, p.mg_maxcy, p.mg_fast = EK_MG_STOP_RESIDUAL, 1e-10, 12, 1
    g = DuctSolver(p, metrics_from_grid(p, xp, yp))
    rng = np.random.default_rng(ny2 * nz2 + nprob)
    kx2 = np.array([(2 * math.pi * (1 + n % 5) / p.lx) ** 2 for n in range(nprob)])
    rhs = rng.standard_normal((nprob, ny2, nz2))
    rhs[:, 0] = rhs[:, -1] = 0
    a, sa, _ = g.multigrid_mudpack(rhs, kx2)
    top = len(g.mg_levels())
    for d in (0, 1):
        g.mg_set_layout(top, d, 16, 8)
    b, sb, _ = g.multigrid_mudpack(rhs, kx2)
    assert sa["max_cycles"] == sb["max_cycles"] and np.isfinite(a).all() and np.array_equal(a, b)
