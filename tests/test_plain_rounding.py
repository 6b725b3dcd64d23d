"""What the plain solver's coarse kernel adds in rounding: problems that it holds
whole, solved until they stand still, are as near their exact solutions as the
oracle's, whose every operation is rounded once in FP64."""
import math

import numpy as np
import pytest

from ekcases import sheared_case, small_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL
from oracle import ekref


def exact(o, kx2, b):
    """Solutions of the oracle's operator (its columns are exact) for the
    right-hand sides b [s][j][k], refined in extended precision."""
    s, ny2, nz2 = b.shape
    n = ny2 * nz2
    eye = np.eye(n)
    a = np.stack([o.mg_apply(kx2, eye[q].reshape(ny2, nz2)).ravel() for q in range(n)], 1)
    al, bl = a.astype(np.longdouble), b.reshape(s, n).T
    x = np.linalg.solve(a, bl).astype(np.longdouble)
    for _ in range(3):
        x = x + np.linalg.solve(a, (bl - al @ x).astype(float))
    return x.T.reshape(b.shape)


@pytest.mark.gpu
@pytest.mark.parametrize("case,ny2,nz2", [(small_case, 33, 9), (sheared_case, 9, 17), (sheared_case, 17, 17),
                                          (sheared_case, 17, 33)])
def test_converged_error_is_the_oracles(case, ny2, nz2):
    p, xp, yp, _ = case(16, ny2, nz2)
    p.mg_stop, p.mg_tol, p.mg_maxcy = EK_MG_STOP_RESIDUAL, 1e-16, 150
    g = DuctSolver(p, metrics_from_grid(p, xp, yp))
    o = ekref.Oracle(p, ekref.metrics_from_grid(p, xp, yp))
    kx2 = np.array([(2 * math.pi * k / p.lx) ** 2 for k in (3, 5, 8)])
    s = 48
    rhs = np.random.default_rng(7).standard_normal((s, 3, ny2, nz2))
    rhs[:, :, 0] = rhs[:, :, -1] = 0
    both = [np.asarray(q.reshape(rhs.shape)) for q in
            (g.multigrid_mudpack(rhs.reshape(-1, ny2, nz2), np.tile(kx2, s))[0],
             o.poisson(rhs.reshape(-1, ny2, nz2), np.tile(kx2, s))[0])]
    x = np.stack([exact(o, k, rhs[:, n]) for n, k in enumerate(kx2)], 1)
    err = [np.sqrt((((q - x) ** 2).sum((2, 3)) / (x ** 2).sum((2, 3))).astype(float)) for q in both]
    mean = [math.exp(np.log(e).mean()) for e in err]
    # means of 144 logarithms, each a few percent from its own expectation
    assert mean[1] < 1e-15 and mean[0] <= 1.15 * mean[1], mean
