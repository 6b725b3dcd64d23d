"""The mixed solver's one-launch levels at the shapes where they differ: a
whole cycle in a block or the finest levels left out, lines of one segment
and of many, a coarsest level in one warp's registers or not (more than 32
points, more than 5 rows), an even number of coarsest columns, orthogonal and
sheared operators.  Against the oracle's operator (the residual the solver
claims) and, bit for bit, against one launch a line solve and transfer."""
import math

import numpy as np
import pytest

from ekcases import sheared_case, small_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL
from oracle import ekref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny2,nz2", [(17, 17), (9, 33), (57, 49), (33, 129), (129, 25), (65, 81), (113, 97)])
@pytest.mark.parametrize("case", [small_case, sheared_case])
def test_one_launch_levels_match_oracle(case, ny2, nz2):
    p, xp, yp, _ = case(16, ny2, nz2)
    p.mg_stop, p.mg_tol, p.mg_maxcy = EK_MG_STOP_RESIDUAL, 1e-10, 200
    o = ekref.Oracle(p, ekref.metrics_from_grid(p, xp, yp))
    q = type(p).from_buffer_copy(p)
    q.mg_fast = 1
    g = DuctSolver(q, metrics_from_grid(p, xp, yp))
    nx, ny = g.mg_levels()[-1]
    assert (nx, ny) == (nz2, ny2) and 0 <= g.mg_tail_levels() <= len(g.mg_levels())
    rng = np.random.default_rng(ny2 * nz2)
    kx2 = np.array([(2 * math.pi * k / p.lx) ** 2 for k in (1, 2, 3, 5)])
    rhs = rng.standard_normal((len(kx2), ny2, nz2))
    rhs[:, 0] = rhs[:, -1] = 0
    a, sa, ca = g.multigrid_mudpack(rhs, kx2)
    assert ca == 0 and sa["max_residual"] <= 1e-10
    for n in range(len(kx2)):
        r = rhs[n] - o.mg_apply(kx2[n], a[n])
        assert np.linalg.norm(r) <= 1.1e-10 * np.linalg.norm(rhs[n]), n
    # the same solve with every level above the Thomas ones in launches of its
    # own: the same operations on the same values
    for lev in range(2, len(g.mg_levels()) + 1):
        for d in (0, 1):
            g.mg_set_layout(lev, d, 16, 8)
    b, sb, _ = g.multigrid_mudpack(rhs, kx2)
    assert sa["max_cycles"] == sb["max_cycles"] and np.array_equal(a, b)
