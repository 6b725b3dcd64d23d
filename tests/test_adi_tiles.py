"""The tiled line solves of the mixed path (increment form, and float-float
with LES) at the sizes where their tiles end: fewer x points than a tile's
32, lines of one row more or less than whole chunks of 8 and 16, one chunk
only.  Against the FP64 oracle at the same 1e-10 residual rule."""
import numpy as np
import pytest

from ekcases import les_case, rel_l2, sheared_case, small_case
from ekman_bl_gb300.duct import DuctSolver, les_metrics_from_grid, metrics_from_grid
from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL
from oracle import ekref

pytestmark = pytest.mark.gpu


def pair(p, xp, yp, st):
    p.mg_stop, p.mg_tol, p.mg_maxcy = EK_MG_STOP_RESIDUAL, 1e-10, 200
    o = ekref.Oracle(p, ekref.metrics_from_grid(p, xp, yp))
    q = type(p).from_buffer_copy(p)
    q.mg_maxcy, q.mg_fast, q.fft_fp32, q.ff_arith = 60, 1, 1, 2
    g = DuctSolver(q, metrics_from_grid(p, xp, yp))
    if p.les:
        o.set_les_metrics(ekref.les_metrics_from_grid(p, xp, yp))
        g.set_les_metrics(les_metrics_from_grid(p, xp, yp))
    g.upload(*st)
    o.upload(*st)
    return g, o


@pytest.mark.parametrize("nx,ny2,nz2", [(8, 17, 25), (16, 9, 33), (32, 25, 17), (64, 41, 57), (16, 33, 9)])
@pytest.mark.parametrize("case", ["small", "sheared", "les"])
def test_tiled_line_solves_track_oracle(case, nx, ny2, nz2):
    make = {"small": small_case, "sheared": sheared_case, "les": lambda *a: les_case("small", nx=a[0], ny2=a[1], nz2=a[2])}
    g, o = pair(*make[case](nx, ny2, nz2))
    g.step(1)
    o.step(1)
    a, b = g.download(), o.download()
    # FP32 increments and products: a few 2^-24 of the fields a substep; a
    # wrong row, neighbour or chunk end shows at the increments' size, 1e-3
    for name, f in zip(("CU1", "CU2", "CU3", "CTH"), (0, 1, 2, 4)):
        e = rel_l2(a[f], b[f])
        assert np.isfinite(e) and e < 1e-5, (name, e)


@pytest.mark.parametrize("nx,ny2,nz2", [(512, 19, 257), (1024, 9, 129)])
def test_one_thread_a_system_tracks_oracle(nx, ny2, nz2):
    """Sweeps of enough lines that the float-float y sweep with LES goes one
    thread a system (rows short of and past whole chunks of 4 and 8)."""
    test_tiled_line_solves_track_oracle("les", nx, ny2, nz2)
