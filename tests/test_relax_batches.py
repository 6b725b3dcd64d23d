"""The plain solver's two ways of relaxing a sheared level, one block a problem
or a launch a phase, at the sizes where the choice between them turns: more
phi than a block's shared memory, and batches just within and beyond the most
that a block a problem takes.  Against the oracle's MUDPACK schedule, and one
way against the other bit for bit: the operations are the same."""
import math

import numpy as np
import pytest

from ekcases import rel_l2, sheared_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from oracle import ekref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny2,nz2,nprob", [(129, 257, 3), (257, 113, 2),   # launches: phi over 220 KB
                                           (161, 161, 457), (193, 129, 457)])  # launches: a fourth wave
def test_relaxation_by_launches(ny2, nz2, nprob):
    p, xp, yp, _ = sheared_case(16, ny2, nz2)
    g = DuctSolver(p, metrics_from_grid(p, xp, yp))
    o = ekref.Oracle(p, ekref.metrics_from_grid(p, xp, yp))
    kx2 = np.array([(2 * math.pi * (1 + k % 5) / p.lx) ** 2 for k in range(nprob)])
    few = 3
    rhs = np.random.default_rng(ny2).standard_normal((few, ny2, nz2))
    rhs[:, 0] = rhs[:, -1] = 0
    idx = np.arange(nprob) % few
    kx2 = kx2[idx]
    a, sa, _ = g.multigrid_mudpack(rhs[idx], kx2)
    b, sb, _ = o.poisson(rhs[:min(few, nprob)], kx2[:min(few, nprob)])
    assert (sa["min_cycles"], sa["max_cycles"]) == (sb["min_cycles"], sb["max_cycles"])
    # as in the one-block form's test: a few thousand dependent updates, each
    # a few 2^-53 of phi, damped by the cycles
    assert rel_l2(a[:few], b) < 1e-12
    assert np.array_equal(a, a[idx])
    if nprob > few:
        # one block a problem
        c, sc, _ = g.multigrid_mudpack(rhs, kx2[:few])
        assert sc["max_cycles"] == sa["max_cycles"] and np.array_equal(c, a[:few])
        c, _, _ = g.multigrid_mudpack(rhs[idx[:456]], kx2[:456])
        assert np.array_equal(c, a[:456])
