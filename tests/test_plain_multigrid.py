"""The plain solver's one-block relaxation and coarse levels at the shapes
where they differ: more points a phase than threads, fewer than a warp, phases
whose points share two lanes or not, orthogonal and sheared operators.
Against the oracle's MUDPACK schedule: the same cycles, the same solutions up
to the order of FP64 sums."""
import math

import numpy as np
import pytest

from ekcases import rel_l2, sheared_case, small_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from oracle import ekref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,ny2,nz2", [(sheared_case, 129, 129), (sheared_case, 17, 33), (sheared_case, 33, 9),
                                          (sheared_case, 49, 41), (small_case, 65, 49), (small_case, 9, 17)])
def test_plain_solve_matches_oracle(case, ny2, nz2):
    p, xp, yp, _ = case(16, ny2, nz2)
    g = DuctSolver(p, metrics_from_grid(p, xp, yp))
    o = ekref.Oracle(p, ekref.metrics_from_grid(p, xp, yp))
    kx2 = np.array([(2 * math.pi * k / p.lx) ** 2 for k in (1, 2, 5)])
    rhs = np.random.default_rng(ny2).standard_normal((3, ny2, nz2))
    rhs[:, 0] = rhs[:, -1] = 0
    a, sa, _ = g.multigrid_mudpack(rhs, kx2)
    b, sb, _ = o.poisson(rhs, kx2)
    assert (sa["min_cycles"], sa["max_cycles"]) == (sb["min_cycles"], sb["max_cycles"])
    # a few thousand dependent updates, each a few 2^-53 of phi, damped by the cycles
    assert rel_l2(a, b) < 1e-12
