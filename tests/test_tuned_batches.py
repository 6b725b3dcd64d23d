"""Tuning on a grid whose own batch is too large for the one-block levels: a
smaller batch solved on the same context keeps them, and its bits."""
import math

import numpy as np
import pytest

from ekcases import small_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL

pytestmark = pytest.mark.gpu


def test_tuning_leaves_small_batches_alone():
    p, xp, yp, st = small_case(nx=256, ny2=65, nz2=65, mg_stop=EK_MG_STOP_RESIDUAL)  # 172 problems a projection
    p.mg_tol, p.mg_maxcy, p.mg_fast = 1e-10, 60, 1
    g = DuctSolver(p, metrics_from_grid(p, xp, yp))
    g.upload(*st)
    rng = np.random.default_rng(2)
    kx2 = np.array([(2 * math.pi * k / p.lx) ** 2 for k in (1, 2, 3, 5, 8, 10)])
    rhs = rng.standard_normal((len(kx2), 65, 65))
    rhs[:, 0] = rhs[:, -1] = 0

    def solve():
        n = g.launch_count()
        phi, s, c = g.multigrid_mudpack(rhs, kx2)
        assert c == 0
        return phi, s["max_cycles"], g.launch_count() - n

    phi0, cyc0, n0 = solve()
    g.mg_autotune(reps=2)
    phi1, cyc1, n1 = solve()
    assert (cyc1, n1) == (cyc0, n0) and np.array_equal(phi0, phi1)
    # by hand, the finest level has launches of its own (in one direction
    # alone, the other takes the tuned layout, whose segments may be shorter),
    # and none again with 0
    top = len(g.mg_levels())
    g.mg_set_layout(top, 0, 16, 8)
    assert solve()[2] > n0
    g.mg_set_layout(top, 1, 16, 8)
    phi2, _, n2 = solve()
    assert n2 > n0 and np.array_equal(phi0, phi2)
    g.mg_set_layout(top, 0, 0, 0)
    assert solve()[2] > n0
    g.mg_set_layout(top, 1, 0, 0)
    phi3, _, n3 = solve()
    assert n3 == n0 and np.array_equal(phi0, phi3)
