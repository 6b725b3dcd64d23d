"""A state that is not finite, in one mode of one field at one point: the first
substep's projection reports it, on orthogonal grids too, whose kernels leave
out the products with zero metrics that would carry it to the neighbours."""
import numpy as np
import pytest

from ekcases import sheared_case, small_case
from ekman_bl_gb300.duct import DuctSolver, EkError, metrics_from_grid
from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL

pytestmark = pytest.mark.gpu

EK_ERR_NAN = 4


@pytest.mark.parametrize("case", [small_case, sheared_case])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_first_substep_reports_it(case, mixed, value):
    p, xp, yp, st = case()
    if mixed:
        p.mg_stop, p.mg_tol, p.mg_maxcy = EK_MG_STOP_RESIDUAL, 1e-8, 20
        p.mg_fast, p.fft_fp32, p.ff_arith = 1, 1, 2
    g = DuctSolver(p, metrics_from_grid(p, xp, yp))
    for f in range(5):
        for j, k in ((1, 1), (3, 4), (p.ny, p.nz)):
            cu = [np.array(a) for a in st]
            cu[f][j, k, 1] = value
            g.upload(*cu)
            with pytest.raises(EkError) as e:
                g.rk_duct(1)
            assert e.value.code == EK_ERR_NAN, (f, j, k)
    # the context is as good as before
    g.upload(*st)
    g.rk_duct(1)
    assert np.isfinite(g.divergence())
