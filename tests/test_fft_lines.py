"""The context-free x-transforms at every size they take, with line counts that
leave a warp's and a block's last lines empty, and cutoffs from the mean mode
alone to all but the last."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [8, 16, 32, 64, 128, 256, 512, 1024])
@pytest.mark.parametrize("lines", [1, 5, 131])
def test_transforms_match_numpy(nx, lines):
    import torch
    from ekman_bl_gb300.duct import fft_x
    rng = np.random.default_rng(nx + lines)
    u = np.zeros((lines, nx + 2))
    u[:, :nx] = rng.standard_normal((lines, nx))
    # an FFT's rounding grows as log2(NX) 2^-53 of the values
    tol = 4 * np.log2(nx) * 2.0 ** -53
    for nkx in (0, nx // 3, nx // 2 - 1):
        d = torch.from_numpy(u).cuda()
        s = torch.full((lines, nx // 2 + 1), 7.0, dtype=torch.complex128, device="cuda")
        fft_x(True, nx, nkx, lines, d.data_ptr(), s.data_ptr())
        ref = np.fft.rfft(u[:, :nx], axis=1) / nx
        ref[:, nkx + 1:] = 0
        a = s.cpu().numpy()
        assert np.all(a[:, nkx + 1:] == 0)
        assert np.linalg.norm(a - ref) <= tol * np.linalg.norm(u) / np.sqrt(nx)
        # the inverse reads modes 0..nkx and ignores the mean's imaginary part
        x = rng.standard_normal((lines, nx // 2 + 1)) + 1j * rng.standard_normal((lines, nx // 2 + 1))
        s = torch.from_numpy(x).cuda()
        d = torch.full((lines, nx + 2), 7.0, dtype=torch.float64, device="cuda")
        fft_x(False, nx, nkx, lines, s.data_ptr(), d.data_ptr())
        y = x.copy()
        y[:, nkx + 1:] = 0
        y[:, 0] = y[:, 0].real
        ref = np.fft.irfft(y, n=nx, axis=1) * nx
        b = d.cpu().numpy()
        assert np.all(b[:, nx:] == 0)
        assert np.linalg.norm(b[:, :nx] - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("nx", [16, 64, 128, 256])
@pytest.mark.parametrize("lines", [701, 709, 1999, 2001])
def test_line_counts_about_the_packing_rule(nx, lines):
    """Both forms on either side of the line count that chooses between them."""
    test_transforms_match_numpy(nx, lines)


@pytest.mark.parametrize("nx", [64, 128, 256, 512, 1024])
@pytest.mark.parametrize("ff", [1, 2])
def test_mixed_step_at_every_transform_size(nx, ff):
    """A mixed-path step, straight and sheared, against the FP64 oracle at the
    mixed path's bar: the transforms' loads in batches at each size."""
    from ekcases import rel_l2, sheared_case, small_case
    from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
    from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL
    from oracle import ekref
    p, xp, yp, st = (sheared_case if nx in (128, 512) else small_case)(nx=nx)
    p.mg_stop, p.mg_tol, p.mg_maxcy = EK_MG_STOP_RESIDUAL, 1e-10, 200
    q = type(p).from_buffer_copy(p)
    q.mg_maxcy, q.mg_fast, q.fft_fp32, q.ff_arith = 60, 1, 1, ff
    m = metrics_from_grid(p, xp, yp)
    g, o = DuctSolver(q, m), ekref.Oracle(p, m)
    try:
        g.upload(*st)
        o.upload(*st)
        g.step(1)
        o.step(1)
        for name, x, y in zip(("CU1", "CU2", "CU3", "CTH"), *[[v[i] for i in (0, 1, 2, 4)] for v in (g.download(), o.download())]):
            assert rel_l2(x, y) < 1e-5, name
    finally:
        g.close()
        o.close()
