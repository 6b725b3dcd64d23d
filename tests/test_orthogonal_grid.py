"""On an orthogonal grid the step leaves out the terms of GMAT_12, CJOB_12 and
CJOB_21.  One nonzero entry of any of the three takes the whole grid back to
the general kernels; minus zero counts as zero."""
import numpy as np
import pytest

from ekcases import rel_l2, small_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL
from oracle import ekref


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name,value", [("gmat_12", -0.0), ("gmat_12", 0.05), ("cjob_12", 0.05), ("cjob_21", 0.05)])
def test_one_cross_metric(name, value, mixed):
    """A step against the FP64 oracle with the bars of the other step tests:
    1e-10 in FP64, 1e-5 on the mixed path.  The entry is `value` of the
    diagonal metrics' mean, large enough to be seen past either bar."""
    p, xp, yp, st = small_case(nx=16)
    p.mg_stop, p.mg_tol, p.mg_maxcy = EK_MG_STOP_RESIDUAL, 1e-12, 200
    m = {k: np.array(v) for k, v in metrics_from_grid(p, xp, yp).items()}
    a = m[name]
    if value < 0 or np.signbit(value):
        a[...] = -0.0
    else:
        a[:, a.shape[1] // 2, a.shape[2] // 2] = value * np.abs(m["gmat_11"]).mean()
    q = type(p).from_buffer_copy(p)
    if mixed:
        q.mg_tol, q.mg_maxcy, q.mg_fast, q.fft_fp32, q.ff_arith = 1e-10, 60, 1, 1, 2
    g, o = DuctSolver(q, m), ekref.Oracle(p, m)
    try:
        g.upload(*st)
        o.upload(*st)
        g.step(1)
        o.step(1)
        for n, x, y in zip(("CU1", "CU2", "CU3", "CTH"), *[[v[i] for i in (0, 1, 2, 4)] for v in (g.download(), o.download())]):
            assert rel_l2(x, y) < (1e-5 if mixed else 1e-10), n
    finally:
        g.close()
        o.close()
