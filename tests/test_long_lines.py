"""Lines of more rows than a tile of the increment form's line solves holds
(1,600): the kernel without tiles, in either direction, against the FP64 oracle
at the same 1e-10 residual rule."""
import numpy as np
import pytest

from ekcases import rel_l2, sheared_case, small_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL
from oracle import ekref

pytestmark = pytest.mark.gpu


def pair(p, xp, yp, st, cycles):
    p.mg_stop, p.mg_tol, p.mg_maxcy = EK_MG_STOP_RESIDUAL, 1e-10, cycles
    o = ekref.Oracle(p, ekref.metrics_from_grid(p, xp, yp))
    q = type(p).from_buffer_copy(p)
    q.mg_fast, q.fft_fp32, q.ff_arith = 1, 1, 2
    g = DuctSolver(q, metrics_from_grid(p, xp, yp))
    g.upload(*st)
    o.upload(*st)
    return g, o


@pytest.mark.parametrize("case,ny2,nz2", [(small_case, 2049, 9), (small_case, 9, 2049), (small_case, 1601, 9),
                                          (sheared_case, 2049, 9), (small_case, 1537, 9)])
def test_lines_beyond_a_tile(case, ny2, nz2):
    g, o = pair(*case(8, ny2, nz2), cycles=60)
    g.rk_duct(1)
    o.rk_substep(1)
    a, b = g.download(), o.download()
    # Point relaxation leaves the kx = 0 problem of such thin grids far from its
    # solution, so its mode is compared for the scalar alone, which no pressure
    # enters.  The bound of the tiled sweeps: FP32 increments and products, a
    # few 2^-24 of the fields a substep.
    for name, f, k0 in (("CU1", 0, 1), ("CU2", 1, 1), ("CU3", 2, 1), ("CTH", 4, 0)):
        e = rel_l2(a[f][..., k0:], b[f][..., k0:])
        assert np.isfinite(e) and e < 1e-5, (name, e)
