"""The CFL step takes a line's largest speed first and divides once: the
binding point at either end of a line, in a line shorter than, equal to and
longer than a warp, for each of the three velocity components."""
import numpy as np
import pytest

from ekcases import cfl_case, sheared_case
from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
from oracle import ekref


@pytest.mark.gpu
@pytest.mark.parametrize("comp", [0, 1, 2])
@pytest.mark.parametrize("nx,end,sheared", [(8, 0, False), (16, 1, True), (32, 1, False), (64, 0, False)])
def test_cfl_step_of_a_spike(nx, end, sheared, comp):
    """A band-limited spike in one component on one (k, j) line near the middle.
    The state agrees with the oracle's to 1e-10 (rel_l2) after a step, so a
    point's speed, and with it DELTA_T, agrees to that as well."""
    p, xp, yp, st = cfl_case(0.2, 1.0, nx=nx)
    if sheared:
        q, xp, yp, st = sheared_case(nx=nx)
        q.variable_dt, q.update_dt, q.cfl, q.delta_t_set = 1, 1, 0.2, 1.0
        p = q
    p.cfl = 1.0
    st = [np.array(a) for a in st]
    u = st[comp]
    x0 = (nx - 1 if end else 0) / nx
    modes = np.arange(nx // 3 + 1)
    u[u.shape[0] // 2, u.shape[1] // 2, : nx // 3 + 1] += 4.0 / nx * np.exp(-2j * np.pi * modes * x0)
    g = DuctSolver(p, metrics_from_grid(p, xp, yp))
    o = ekref.Oracle(p, ekref.metrics_from_grid(p, xp, yp))
    try:
        g.upload(*st)
        o.upload(*st)
        g.step(1)
        o.step(1)
        dg, do = g.get_time()[2], o.get_time()[2]
        assert do < 1.0 and abs(dg - do) <= 1e-10 * do
    finally:
        g.close()
        o.close()
