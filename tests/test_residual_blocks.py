"""The mixed solver's residual and its per-problem decision: rows cut into
several blocks' runs (short and empty ones among them) or not, the decision in
the residual's last block or in a launch of its own, problem counts that leave
lanes empty.  Each solution against the oracle's operator at the residual the
solver claims, and the cap on the cycles."""
import math

import numpy as np
import pytest

from ekcases import sheared_case, small_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL
from oracle import ekref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,ny2,nz2,nprob", [
    (small_case, 17, 17, 1), (small_case, 17, 129, 33), (sheared_case, 33, 49, 100),
    (small_case, 129, 65, 128), (sheared_case, 129, 33, 150), (small_case, 65, 65, 300)])
def test_residual_and_decision(case, ny2, nz2, nprob):
    p, xp, yp, _ = case(16, ny2, nz2)
    p.mg_stop, p.mg_tol, p.mg_maxcy = EK_MG_STOP_RESIDUAL, 1e-10, 200
    o = ekref.Oracle(p, ekref.metrics_from_grid(p, xp, yp))
    q = type(p).from_buffer_copy(p)
    q.mg_fast = 1
    g = DuctSolver(q, metrics_from_grid(p, xp, yp))
    rng = np.random.default_rng(ny2 * nz2 + nprob)
    kx2 = np.array([(2 * math.pi * (1 + n % 7) / p.lx) ** 2 for n in range(nprob)])
    rhs = rng.standard_normal((nprob, ny2, nz2))
    rhs[:, 0] = rhs[:, -1] = 0
    a, sa, ca = g.multigrid_mudpack(rhs, kx2)
    assert ca == 0 and sa["max_residual"] <= 1e-10
    for n in sorted({0, 1 % nprob, nprob // 2, nprob - 1}):
        r = rhs[n] - o.mg_apply(kx2[n], a[n])
        assert np.linalg.norm(r) <= 1.1e-10 * np.linalg.norm(rhs[n]), n
    # stopped at one cycle, every problem is reported
    q.mg_maxcy = 1
    h = DuctSolver(q, metrics_from_grid(p, xp, yp))
    _, sb, _ = h.multigrid_mudpack(rhs, kx2)
    assert sb["min_cycles"] == sb["max_cycles"] == 1 and sb["n_not_converged"] == nprob
