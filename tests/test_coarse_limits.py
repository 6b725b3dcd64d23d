"""Plain solves on grids whose coarsest level alone fills a block's shared
memory (sides of 53, 43 and 45 times two, plus one): against the oracle."""
import math

import numpy as np
import pytest

from ekcases import rel_l2, sheared_case, small_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from oracle import ekref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,ny2,nz2,level1", [(small_case, 107, 107, (54, 54)), (small_case, 107, 111, (56, 54)),
                                                 (sheared_case, 87, 91, (46, 44)), (small_case, 87, 91, (46, 44))])
def test_large_coarsest_level(case, ny2, nz2, level1):
    p, xp, yp, _ = case(16, ny2, nz2)
    g = DuctSolver(p, metrics_from_grid(p, xp, yp))
    assert g.mg_levels()[0] == level1
    o = ekref.Oracle(p, ekref.metrics_from_grid(p, xp, yp))
    kx2 = np.array([(2 * math.pi * k / p.lx) ** 2 for k in (1, 2, 5)])
    rhs = np.random.default_rng(ny2).standard_normal((3, ny2, nz2))
    rhs[:, 0] = rhs[:, -1] = 0
    a, sa, _ = g.multigrid_mudpack(rhs, kx2)
    b, sb, _ = o.poisson(rhs, kx2)
    assert (sa["min_cycles"], sa["max_cycles"]) == (sb["min_cycles"], sb["max_cycles"])
    # a few thousand dependent updates, each a few 2^-53 of phi, damped by the cycles
    assert rel_l2(a, b) < 1e-12
