"""The work a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values.  Five kinds:

  step      a run between two saves: the state goes in from pinned host
            memory (a restart), `steps` RK3 steps, the state comes back.
            method "mixed" is the mixed-precision path (FP32 V-cycles around a
            float-float residual, FP32 increments), "plain" the FP64 path
            with MUDPACK's own stopping rule (the Fortran driver's drop-in).
            Options: les (dynamic Smagorinsky), cfl (VARIABLE_DT), grid
            "straight" or "sheared" (a non-orthogonal y-z grid).
  ensemble  the same for several runs of uneven sizes stepped together.
  poisson   the batched per-kx Poisson solve on device arrays.
  fft       the context-free batched x-transforms on device arrays.
  unet      the learned guess's network: its prediction, or the prediction,
            loss and parameter gradient of a training batch.

Sizes are NX, NY+2 and NZ+2 as everywhere in this repository.
"""
import math

import numpy as np
import torch

STRETCH = 1.8          # tanh clustering of y at the wall
CELL = 0.3             # y-z cell size in Ekman depths
NOISE = 0.08           # rms of the noise on each velocity and on the scalar
MG_TOL = 1e-8


# ----------------------------------------------------------------------------
# cases
def listed():
    return [
        # the benchmark's workload: the large stratified Ekman layer, the mixed method
        dict(name="step_512x385x257", kind="step", method="mixed", nx=512, ny2=385, nz2=257, steps=4, les=False,
             cfl=False, grid="straight"),
        # the small neutral-case size: short kernels, so launches and latency count
        dict(name="step_64x65x65", kind="step", method="mixed", nx=64, ny2=65, nz2=65, steps=10, les=False,
             cfl=False, grid="straight"),
        # the plain FP64 path on the middle workload, MUDPACK's own stopping rule
        dict(name="step_plain_256x257x193", kind="step", method="plain", nx=256, ny2=257, nz2=193, steps=1, les=False,
             cfl=False, grid="straight"),
        # large-eddy simulation over one C_DYN period (five steps)
        dict(name="step_les_256x193x129", kind="step", method="mixed", nx=256, ny2=193, nz2=129, steps=5, les=True,
             cfl=False, grid="straight"),
        # a curvilinear grid under VARIABLE_DT: the step size follows the CFL number
        dict(name="step_cfl_128x129x97_sheared", kind="step", method="mixed", nx=128, ny2=129, nz2=97, steps=4,
             les=False, cfl=True, grid="sheared"),
        # four runs of uneven sizes advanced together
        dict(name="ensemble_4", kind="ensemble", members=4, sizes=3, lo=64, hi=160, steps=2),
        # every Poisson problem of the large workload, real and imaginary parts, to 1e-8
        dict(name="poisson_512x385x257", kind="poisson", method="mixed", nx=512, ny2=385, nz2=257, grid="straight"),
        # MUDPACK's own cycles on a sheared grid of the middle size (the general smoother)
        dict(name="poisson_plain_64x129x97_sheared", kind="poisson", method="plain", nx=64, ny2=129, nz2=97,
             grid="sheared"),
        # one field of the large workload to Fourier space, and a small one back
        dict(name="fft_forward_512x385x257", kind="fft", forward=True, nx=512, lines=385 * 257),
        dict(name="fft_inverse_64x65x65", kind="fft", forward=False, nx=64, lines=65 * 65),
        # a training batch of the learned guess on the large workload's images
        dict(name="unet_gradient_16x72x104", kind="unet", gradient=True, channels=32, n=16, h=72, w=104),
    ]


def _mudpack_sizes(hi):
    """Sides MUDPACK takes, p*2^k + 1 with 2 <= p <= 8, up to hi."""
    return sorted({p * 2 ** k + 1 for p in range(2, 9) for k in range(1, 9) if 17 <= p * 2 ** k + 1 <= hi})


def _side(rng, hi):
    s = _mudpack_sizes(hi)
    v = math.exp(rng.uniform(math.log(16), math.log(hi + 1)))
    return min(s, key=lambda n: (abs(math.log(n / v)), n))


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["poisson"] * 2 + ["fft"] * 2 + ["ensemble", "unet"])
    if kind == "step":
        method = rng.choice(["mixed", "mixed", "plain"])
        les, cfl = rng.random() < 0.25, rng.random() < 0.2
        grid = rng.choice(["straight", "straight", "sheared"])
        while True:
            nx, ny2, nz2 = rng.choice([32, 64, 128, 256, 512]), _side(rng, 385), _side(rng, 257)
            steps = rng.randint(1, 5)
            cost = nx * ny2 * nz2 * steps * (3 if method == "plain" else 1) * (2 if les else 1)
            if cost <= 0.75 * 512 * 385 * 257:
                return dict(kind=kind, method=method, nx=nx, ny2=ny2, nz2=nz2, steps=steps, les=les, cfl=cfl, grid=grid)
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(2, 6), sizes=rng.randint(0, 10 ** 6), lo=32, hi=160,
                    steps=rng.randint(1, 3))
    if kind == "poisson":
        method = rng.choice(["mixed", "mixed", "plain"])
        hi = 1 if method == "mixed" else 4
        while True:
            nx, ny2, nz2 = rng.choice([16, 32, 64, 128, 256, 512]), _side(rng, 385), _side(rng, 257)
            if nx * ny2 * nz2 * hi <= 512 * 385 * 257:
                return dict(kind=kind, method=method, nx=nx, ny2=ny2, nz2=nz2, grid=rng.choice(["straight", "sheared"]))
    if kind == "fft":
        nx = rng.choice([16, 32, 64, 128, 256, 512, 1024])
        most = 512 * 385 * 257 // nx
        return dict(kind=kind, forward=rng.random() < 0.5, nx=nx,
                    lines=int(math.exp(rng.uniform(math.log(257), math.log(most)))))
    return dict(kind=kind, gradient=rng.random() < 0.5, channels=rng.choice([16, 32]), n=rng.randint(4, 48),
                h=8 * rng.randint(3, 12), w=8 * rng.randint(3, 14))


# ----------------------------------------------------------------------------
# inputs
def _depth(nu):
    return math.sqrt(2.0 * nu)      # Ekman depth for f = 1


def _grid(ny2, nz2, nu, grid):
    """xpoint, ypoint [J, K]: uniform streamwise z, y clustered at the wall;
    sheared: the streamwise points move with height."""
    h = CELL * _depth(nu)
    j = np.arange(ny2)[:, None]
    y = (ny2 - 1) * h * (1.0 + np.tanh(STRETCH * (j / (ny2 - 1) - 1.0)) / math.tanh(STRETCH))
    x = np.arange(nz2)[None, :] * h
    if grid == "sheared":
        x = x + 0.3 * h * np.sin(2.0 * math.pi * j / (ny2 - 1))
    return (np.ascontiguousarray(np.broadcast_to(x, (ny2, nz2))), np.ascontiguousarray(np.broadcast_to(y, (ny2, nz2))))


NU = 2.0e-6             # Re = 1000 on the Ekman depth


def _params(method, nx, ny2, nz2, les=False, cfl=False):
    from ekman_bl_gb300.params import EK_MG_STOP_RESIDUAL, default_params
    p = default_params(nx, ny2 - 2, nz2 - 2)
    p.nu, p.pr, p.ri_tau = NU, 0.7, 0.1
    p.delta_t = p.delta_t_set = 3.0e-4
    p.lx = 0.25 * nx * _depth(NU)
    if method == "mixed":
        p.mg_fast, p.fft_fp32, p.ff_arith = 1, 1, 2
        p.mg_stop, p.mg_tol, p.mg_maxcy = EK_MG_STOP_RESIDUAL, MG_TOL, 100
    if les:
        p.les, p.create_new_flow = 1, 0
    if cfl:
        p.variable_dt, p.update_dt, p.cfl = 1, 1, 0.6
    return p


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _flow(ny2, nz2, nx, ypoint, gen):
    """An Ekman spiral in kx = 0 plus noise on kx = 1..NX/3 of the velocities
    and the scalar: CU1X, CU2X, CU3X, CPX, CTHX in pinned host memory."""
    eta = torch.from_numpy(ypoint / _depth(NU)).cuda()
    nkx = nx // 3
    out = []
    for f in range(5):
        a = torch.zeros((ny2, nz2, nx // 2 + 1), dtype=torch.complex128, device="cuda")
        if f == 0:
            a[:, :, 0] = torch.exp(-eta) * torch.sin(eta)
        if f == 2:
            a[:, :, 0] = 1.0 - torch.exp(-eta) * torch.cos(eta)
        if f != 3:
            noise = torch.randn((ny2 - 2, nz2 - 2, nkx), dtype=torch.complex128, device="cuda", generator=gen)
            a[1:-1, 1:-1, 1:nkx + 1] = NOISE / math.sqrt(2.0 * nkx) * noise
            del noise
        h = torch.empty(a.shape, dtype=a.dtype, pin_memory=True)
        h.copy_(a)
        out.append(h.numpy())
        del a
    return out


class _Run:
    """One simulation: its solver, the saved state it starts from, and the
    host arrays its result goes to."""

    def __init__(self, p, grid, seed):
        from ekman_bl_gb300.duct import DuctSolver, les_metrics_from_grid, metrics_from_grid
        ny2, nz2 = p.ny + 2, p.nz + 2
        xp, yp = _grid(ny2, nz2, NU, grid)
        self.p = p
        self.solver = DuctSolver(p, metrics_from_grid(p, xp, yp))
        if p.les:
            self.solver.set_les_metrics(les_metrics_from_grid(p, xp, yp))
        self.state = _flow(ny2, nz2, p.nx, yp, _generator(seed))
        torch.cuda.synchronize()
        self.out = [torch.empty(a.shape, dtype=torch.complex128, pin_memory=True).numpy() for a in self.state]
        # the saved state is divergence-free, as CREATE_FLOW leaves it
        self.solver.upload(*self.state)
        self.solver.rem_div_curv()
        self.solver.download(out=self.state)

    def load(self):
        self.solver.upload(*self.state)
        self.solver.set_time(0.0, 0)
        if self.p.les:
            self.solver.les_set_first_time(True)

    def save(self):
        return self.solver.download(out=self.out)


def _ensemble_sizes(case):
    """(NX, NY+2, NZ+2) of the members."""
    rng = np.random.default_rng(case["sizes"])
    sides = [n for n in _mudpack_sizes(2 * case["hi"]) if case["lo"] < n <= case["hi"] + 1]
    return [(int(rng.choice([32, 64, 128])), int(rng.choice(sides)), int(rng.choice(sides)))
            for _ in range(case["members"])]


def _poisson_kx2(nx):
    lx = 0.25 * nx * _depth(NU)
    return np.array([(2.0 * math.pi * (q // 2) / lx) ** 2 for q in range(2 * (nx // 3 + 1))])


def _poisson_rhs(nx, ny2, nz2, seed):
    rhs = torch.randn((2 * (nx // 3 + 1), ny2, nz2), dtype=torch.float64, device="cuda", generator=_generator(seed))
    rhs[:, 0, :] = rhs[:, -1, :] = 0
    rhs[:, :, 0] = rhs[:, :, -1] = 0
    return rhs


def _fft_input(case, seed):
    nx, lines, gen = case["nx"], case["lines"], _generator(seed)
    if case["forward"]:
        a = torch.randn((lines, nx + 2), dtype=torch.float64, device="cuda", generator=gen)
        a[:, nx:] = 0
        return a
    a = torch.zeros((lines, nx // 2 + 1), dtype=torch.complex128, device="cuda")
    nkx = nx // 3
    a[:, :nkx + 1] = torch.randn((lines, nkx + 1), dtype=torch.complex128, device="cuda", generator=gen)
    a[:, 0].imag.zero_()
    return a


def _unet_layers(c):
    return [(2, c)] + [(c, c)] * 7 + [(2 * c, c), (c, c)] * 3 + [(c, 1)]


def _unet_input(case, seed):
    """Images as the solver makes them: a rough right-hand side of unit size
    and a wavenumber channel, a smooth target, zero outside the valid part."""
    n, h, w, gen = case["n"], case["h"], case["w"], _generator(seed)
    hv, wv = h - 3, w - 5
    x = torch.zeros((n, h, w, 2), device="cuda")
    x[:, :hv, :wv, 0] = torch.randn((n, hv, wv), device="cuda", generator=gen)
    x[:, :hv, :wv, 1] = (torch.rand((n, 1, 1), device="cuda", generator=gen) * 0.8 +
                         0.1 * torch.linspace(0, 1, hv, device="cuda")[None, :, None])
    t = torch.zeros((n, h, w), device="cuda")
    s = torch.nn.functional.avg_pool2d(torch.randn((n, 1, hv, wv), device="cuda", generator=gen), 9, 1, 4)[:, 0]
    t[:, :hv, :wv] = s / s.square().mean((1, 2), keepdim=True).sqrt()
    params = []
    for ci, co in _unet_layers(case["channels"]):
        params.append(torch.randn(co * 9 * ci, device="cuda", generator=gen) * math.sqrt(2.0 / (9 * ci)))
        params.append(0.05 * torch.randn(co, device="cuda", generator=gen))
    return x, t, torch.cat(params).cpu().numpy(), hv, wv


# ----------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        p = _params(case["method"], case["nx"], case["ny2"], case["nz2"], case["les"], case["cfl"])
        return {"kind": kind, "steps": case["steps"], "run": _Run(p, case["grid"], seed)}
    if kind == "ensemble":
        runs = [_Run(_params("mixed", *s), "straight", seed + 1000 * m) for m, s in enumerate(_ensemble_sizes(case))]
        return {"kind": kind, "steps": case["steps"], "runs": runs}
    if kind == "poisson":
        from ekman_bl_gb300.duct import DuctSolver, metrics_from_grid
        nx, ny2, nz2 = case["nx"], case["ny2"], case["nz2"]
        p = _params(case["method"], nx, ny2, nz2)
        solver = DuctSolver(p, metrics_from_grid(p, *_grid(ny2, nz2, NU, case["grid"])))
        rhs = _poisson_rhs(nx, ny2, nz2, seed)
        st = {"kind": kind, "solver": solver, "rhs": rhs, "phi": torch.zeros_like(rhs),
              "kx2": torch.from_numpy(_poisson_kx2(nx)).cuda()}
        torch.cuda.synchronize()
        return st
    if kind == "fft":
        a = _fft_input(case, seed)
        nx, lines = case["nx"], case["lines"]
        out = (torch.empty((lines, nx // 2 + 1), dtype=torch.complex128, device="cuda") if case["forward"] else
               torch.empty((lines, nx + 2), dtype=torch.float64, device="cuda"))
        return {"kind": kind, "forward": case["forward"], "nx": nx, "lines": lines, "in": a, "out": out}
    from ekman_bl_gb300.duct import UNet
    x, t, params, hv, wv = _unet_input(case, seed)
    net = UNet(2, case["channels"], case["n"], case["h"], case["w"])
    net.set_params(params)
    torch.cuda.synchronize()
    return {"kind": kind, "gradient": case["gradient"], "net": net, "x": x, "t": t, "n": case["n"], "hv": hv, "wv": wv,
            "y": torch.empty(t.shape, device="cuda")}


def run(state):
    kind = state["kind"]
    if kind == "step":
        r = state["run"]
        r.load()
        r.solver.step(state["steps"])
        out = r.save()
        if r.p.variable_dt:
            return list(out) + [r.solver.get_time()[2]]
        return list(out)
    if kind == "ensemble":
        from ekman_bl_gb300.duct import ensemble_step
        for r in state["runs"]:
            r.load()
        ensemble_step([r.solver for r in state["runs"]], state["steps"])
        return [r.save() for r in state["runs"]]
    if kind == "poisson":
        rhs, phi, kx2 = state["rhs"], state["phi"], state["kx2"]
        state["solver"].multigrid_mudpack_device(rhs.data_ptr(), phi.data_ptr(), kx2.data_ptr(), rhs.shape[0])
        return [phi[:2], phi[2:]]
    if kind == "fft":
        from ekman_bl_gb300.duct import fft_x
        nx, a, out = state["nx"], state["in"], state["out"]
        fft_x(state["forward"], nx, nx // 3, state["lines"], a.data_ptr(), out.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
        return out
    net, x, t, y, n = state["net"], state["x"], state["t"], state["y"], state["n"]
    stream = torch.cuda.current_stream().cuda_stream
    if state["gradient"]:
        loss, grad = net.gradient(x.data_ptr(), t.data_ptr(), n, state["hv"], state["wv"], y.data_ptr(), stream)
        return [float(loss), grad, y]
    net.forward(x.data_ptr(), n, y.data_ptr(), stream)
    return y


# ----------------------------------------------------------------------------
def _step_work(nx, ny2, nz2, steps, les):
    """The state once in and once out; per substep and point 17 x-transforms
    (4 more with LES) of 2.5 log2 NX operations, about 300 operations of
    stencils, line solves and projection, and five corrections of the
    Poisson problems at about 80 operations a point with the coarse levels."""
    pts = nx * ny2 * nz2
    state = 5 * 16.0 * (nx // 2 + 1) * ny2 * nz2
    modes = 2.0 * (nx // 3 + 1) / nx
    per = (21 if les else 17) * 2.5 * math.log2(nx) + (500 if les else 300) + 5 * 80 * 4 / 3 * modes
    return {"bytes": 2 * state, "flops": 3.0 * steps * pts * per}


def work(case):
    kind = case["kind"]
    if kind == "step":
        return _step_work(case["nx"], case["ny2"], case["nz2"], case["steps"], case["les"])
    if kind == "ensemble":
        ws = [_step_work(*s, case["steps"], False) for s in _ensemble_sizes(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if kind == "poisson":
        n = 2 * (case["nx"] // 3 + 1) * case["ny2"] * case["nz2"]
        return {"bytes": 16.0 * n, "flops": 5 * 80 * 4 / 3 * n}
    if kind == "fft":
        nx, lines = case["nx"], case["lines"]
        spectral = 16.0 * ((nx // 2 + 1) if case["forward"] else (nx // 3 + 1))
        return {"bytes": lines * (8.0 * (nx + 2) + spectral), "flops": lines * 2.5 * nx * math.log2(nx)}
    n, h, w, c = case["n"], case["h"], case["w"], case["channels"]
    mult = [(0, 2, c), (0, c, c), (1, c, c), (1, c, c), (2, c, c), (2, c, c), (3, c, c), (3, c, c),
            (2, 2 * c, c), (2, c, c), (1, 2 * c, c), (1, c, c), (0, 2 * c, c), (0, c, c), (0, c, 1)]
    flops = sum(2.0 * 9 * ci * co * n * h * w / 4 ** lv for lv, ci, co in mult)
    npar = sum(9 * ci * co + co for ci, co in _unet_layers(c))
    if case["gradient"]:
        return {"bytes": 4.0 * (4 * n * h * w + 2 * npar), "flops": 3 * flops}
    return {"bytes": 4.0 * (3 * n * h * w + npar), "flops": flops}


# ----------------------------------------------------------------------------
# the same results in 64 bits, from plain numpy and torch
def _metrics(xp, yp):
    """GMAT_11, GMAT_12, GMAT_22 [f, J, K] and INT_JACOB [J, K] of a grid, as
    JACOBI_TRANS forms them (face derivatives cut to 1e-8)."""
    ny, nz = xp.shape[0] - 2, xp.shape[1] - 2
    d = {}
    for name, a in (("x", xp), ("y", yp)):
        z, e = np.zeros((2, ny + 2, nz + 2)), np.zeros((2, ny + 2, nz + 2))
        j, k = slice(1, ny + 1), slice(1, nz + 1)
        jp, kp, jm, km = slice(2, ny + 2), slice(2, nz + 2), slice(0, ny), slice(0, nz)
        z[0, j, k] = a[j, kp] - a[j, k]
        z[1, j, k] = 0.25 * (a[jp, kp] + a[j, kp] - a[jp, km] - a[j, km])
        e[1, j, k] = a[jp, k] - a[j, k]
        e[0, j, k] = 0.25 * (a[jp, k] + a[jp, kp] - a[jm, k] - a[jm, kp])
        e[0, 1] = 2 * e[0, 2] - e[0, 3]
        for q in (e, z):
            q[:, ny + 1] = 2 * q[:, ny] - q[:, ny - 1]
        z[1, 1:, 1] = 2 * z[1, 1:, 2] - z[1, 1:, 3]
        for q in (z, e):
            q[:, 1:, nz + 1] = 2 * q[:, 1:, nz] - q[:, 1:, nz - 1]
        d[name] = [np.trunc(q[:, 1:, 1:] * 1e8) * 1e-8 for q in (z, e)]
    (xz, xe), (yz, ye) = d["x"], d["y"]
    ij = xz * ye - xe * yz
    zx, ex, zy, ey = ye / ij, -yz / ij, -xe / ij, xz / ij
    gs = []
    for v in ((zx * zx + zy * zy) * ij, (zx * ex + zy * ey) * ij, (ex * ex + ey * ey) * ij):
        g = np.zeros((2, ny + 3, nz + 3))
        g[:, 1:ny + 2, 1:nz + 2] = v
        k = slice(0, nz + 2)
        g[:, :ny + 2, 0] = 2 * g[:, :ny + 2, 1] - g[:, :ny + 2, 2]
        g[:, 0, k] = 2 * g[:, 1, k] - g[:, 2, k]
        gs.append(g)
    for g in (gs[0], gs[2]):
        g[:, 0, 0] = 0.5 * (2 * g[:, 1, 0] - g[:, 2, 0] + 2 * g[:, 0, 1] - g[:, 0, 2])
    for g in gs:
        g[:, ny + 2, :nz + 2] = g[:, ny + 1, :nz + 2]
        g[:, :, nz + 2] = g[:, :, nz + 1]
    jac = np.zeros((ny + 2, nz + 2))
    p = np.zeros((2, ny + 3, nz + 3))
    p[:, 1:ny + 2, 1:nz + 2] = ij
    j, k = slice(1, ny + 1), slice(1, nz + 1)
    jac[j, k] = 0.25 * (p[0, j, k] + p[1, j, k] + p[0, 2:ny + 2, k] + p[1, j, 2:nz + 2])
    jac[:, nz + 1], jac[:, 0] = 2 * jac[:, nz] - jac[:, nz - 1], 2 * jac[:, 1] - jac[:, 2]
    jac[ny + 1], jac[0] = 2 * jac[ny] - jac[ny - 1], 2 * jac[1] - jac[2]
    jac[0, 0] = 0.5 * (2 * jac[0, 1] - jac[0, 2] + 2 * jac[1, 0] - jac[2, 0])
    jac[-1, -1] = 0.5 * (2 * jac[-1, -2] - jac[-1, -3] + 2 * jac[-2, -1] - jac[-3, -1])
    return gs, jac


def _operator(xp, yp):
    """The nine-point operator on (NY+2) x (NZ+2) points, periodic in z (the
    first and last column are one place) and Neumann in y: {(dj, di): c[J, K]}
    without the -kx^2 J term, and J."""
    (g11, g12, g22), jac = _metrics(xp, yp)
    ny2, nz2 = jac.shape
    j, k, jp, kp = slice(0, ny2), slice(0, nz2), slice(1, ny2 + 1), slice(1, nz2 + 1)
    around = lambda g: g[1, j, k] + g[1, j, kp] + g[0, j, k] + g[0, jp, k]  # noqa: E731
    cxx, cxy, cyy = 0.25 * around(g11), 0.5 * around(g12), 0.25 * around(g22)
    cx = g11[1, j, kp] - g11[1, j, k] + g12[0, jp, k] - g12[0, j, k]
    cy = g22[0, jp, k] - g22[0, j, k] + g12[1, j, kp] - g12[1, j, k]
    cxx, cyy = np.maximum(cxx, 0.5 * np.abs(cx)), np.maximum(cyy, 0.5 * np.abs(cy))
    c = {(0, 1): cxx + cx / 2, (1, 1): cxy / 4, (1, 0): cyy + cy / 2, (1, -1): -cxy / 4, (0, -1): cxx - cx / 2,
         (-1, -1): cxy / 4, (-1, 0): cyy - cy / 2, (-1, 1): -cxy / 4}
    c[0, 0] = -(c[0, 1] + c[1, 0] + c[0, -1] + c[-1, 0])
    # corners: the diagonal across the corner is taken out, as MUDPACK does
    for jj, ii, s, keep in ((0, 0, -1, ((1, -1), (-1, 1))), (0, nz2 - 1, 1, ((1, 1), (-1, -1))),
                            (ny2 - 1, 0, 1, ((1, 1), (-1, -1))), (ny2 - 1, nz2 - 1, -1, ((1, -1), (-1, 1)))):
        v = s * cxy[jj, ii] / 2
        for o in ((0, 1), (1, 0), (0, -1), (-1, 0)):
            c[o][jj, ii] -= v
        for o in ((1, 1), (1, -1), (-1, 1), (-1, -1)):
            c[o][jj, ii] = v if o in keep else 0.0
        c[0, 0][jj, ii] += 2 * v
    # Neumann rows: what points across the wall folds back onto the mirror row
    for jj, s in ((0, 1), (ny2 - 1, -1)):
        for di in (-1, 0, 1):
            c[s, di][jj] += c[-s, di][jj]
            c[-s, di][jj] = 0.0
    return c, jac


def _poisson_exact(case, seed):
    nx, ny2, nz2 = case["nx"], case["ny2"], case["nz2"]
    modes = nx // 3
    if modes * ny2 * nz2 ** 3 > 32 * 129 * 97 ** 3 or modes * ny2 * nz2 ** 2 > 1.2e9:
        return None                     # over about 20 seconds
    op, jac = _operator(*_grid(ny2, nz2, NU, case["grid"]))
    op, jac = {o: torch.from_numpy(v).cuda() for o, v in op.items()}, torch.from_numpy(jac).cuda()
    rhs = _poisson_rhs(nx, ny2, nz2, seed)
    kx2 = torch.from_numpy(_poisson_kx2(nx)).cuda()[2::2]
    left, right = (torch.arange(nz2, device="cuda") + s for s in (-1, 1))
    left[0], right[-1] = nz2 - 2, 1
    at = torch.arange(nz2, device="cuda")

    def block(j, dj):
        b = torch.zeros((nz2, nz2), dtype=torch.float64, device="cuda")
        for di, col in ((-1, left), (0, at), (1, right)):
            b[at, col] += op[dj, di][j]
        return b

    b = rhs[2:].reshape(modes, 2, ny2, nz2)
    # block elimination down the rows: x_j = d_j - e_j x_{j+1}
    ds, es = [], []
    for j in range(ny2):
        a = block(j, 0) - torch.diag_embed(kx2[:, None] * jac[j])
        v = b[:, :, j].transpose(1, 2)
        if j:
            lo = block(j, -1)
            a, v = a - lo @ es[-1], v - lo @ ds[-1]
        s = torch.linalg.solve(a, torch.cat([v, block(j, 1).expand(modes, -1, -1)], 2))
        ds.append(s[:, :, :2].contiguous())
        es.append(s[:, :, 2:].contiguous())
    x = torch.empty_like(b)
    prev = None
    for j in reversed(range(ny2)):
        prev = ds[j] if prev is None else ds[j] - es[j] @ prev
        x[:, :, j] = prev.transpose(1, 2)
    # the kx = 0 problem is singular: its solution is fixed by convention only
    return [None, x.reshape(2 * modes, ny2, nz2)]


def _fft_exact(case, seed):
    a, nx = _fft_input(case, seed), case["nx"]
    nkx = nx // 3
    if case["forward"]:
        s = torch.fft.rfft(a[:, :nx], dim=1) / nx
        s[:, nkx + 1:] = 0
        return s
    out = torch.zeros((case["lines"], nx + 2), dtype=torch.float64, device="cuda")
    out[:, :nx] = torch.fft.irfft(a, n=nx, dim=1) * nx
    return out


def _unet_exact(case, seed):
    x, t, params, hv, wv = _unet_input(case, seed)
    flat = torch.from_numpy(params).cuda().double().requires_grad_(case["gradient"])
    ws, at = [], 0
    for ci, co in _unet_layers(case["channels"]):
        n = co * 9 * ci
        ws.append((flat[at:at + n].reshape(co, 3, 3, ci).permute(0, 3, 1, 2), flat[at + n:at + n + co]))
        at += n + co
    f = torch.nn.functional
    conv = lambda i, v: f.conv2d(v, ws[i][0], ws[i][1], padding=1)  # noqa: E731
    relu = lambda i, v: torch.relu(conv(i, v))  # noqa: E731
    v = relu(1, relu(0, x.double().permute(0, 3, 1, 2)))
    skips = [v]
    for lv in range(1, 4):
        v = relu(2 * lv + 1, relu(2 * lv, f.avg_pool2d(v, 2)))
        skips.append(v)
    for n, lv in enumerate((2, 1, 0)):
        v = torch.cat([f.interpolate(v, scale_factor=2, mode="nearest"), skips[lv]], 1)
        v = relu(9 + 2 * n, relu(8 + 2 * n, v))
    y = conv(14, v)[:, 0]
    if not case["gradient"]:
        return y
    loss = (y - t.double())[:, :hv, :wv].square().mean()
    loss.backward()
    return [float(loss), flat.grad, y.detach()]


def exact(case, seed):
    """What run() returns for these inputs in 64 bits; None for whole steps
    and ensembles, which take minutes outside this library."""
    if case["kind"] == "poisson":
        return _poisson_exact(case, seed)
    if case["kind"] == "fft":
        return _fft_exact(case, seed)
    if case["kind"] == "unet":
        return _unet_exact(case, seed)
    return None
