"""The work that is timed: time steps, solves and gradients as programs call them.

A case is one of five kinds:

  step      time steps of one grid (les_step, or les_step_io with host fields)
  ensemble  time steps of many ragged grids in one launch
  adjoint   forward and backward of the time-averaged objective
  calls     the step's physics call by call, as a host loop drives it
  pcg       one IC(0)-PCG solve of a matrix that the caller installs

Fields start as the configurations start them: u = 1 + noise, v = w = noise,
p = 0, boundary conditions applied, a cube obstacle, the matrix assembled
before the mask.  Mixed-precision solves run to the relative residual 1e-12
of the adjoint and of the converged comparison trajectories, so that their
result is the discrete solution; FP64 solves run to the configurations' 1e-8.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "les-model_gb300", "py"))
import les_gb300 as G  # noqa: E402

NU, RHO, CS = 1e-5, 1.2, 0.17
CFL_CONV, CFL_VISC, DT_MAX = 0.3, 0.2, 1e-4
NOISE = 0.01
MIXED_TOL, FP64_TOL = 1e-12, 1e-8
PRECOND = {"jacobi": G.PC_JACOBI, "ic": G.PC_IC, "chebyshev": G.PC_CHEBYSHEV}
SOLVER = {"pcg": G.SOLVER_PCG, "jacobi": G.SOLVER_JACOBI, "gs": G.SOLVER_GS}


def _grid(nx, ny, nz, dx, dy=None, dz=None):
    return {"nx": nx, "ny": ny, "nz": nz, "dx": dx, "dy": dy or dx, "dz": dz or dx}


def listed():
    return [
        # the small configuration, FP64 as in the reference: launches and latency count
        dict(name="step_fp64_small", kind="step", steps=2, solver="pcg", mixed=False, precond="jacobi", degree=4,
             **_grid(64, 32, 32, 1 / 32)),
        # the same grid on the mixed path: an interactive or control loop on a small domain
        dict(name="step_mixed_small", kind="step", steps=4, solver="pcg", mixed=True, precond="chebyshev", degree=4,
             **_grid(64, 32, 32, 1 / 32)),
        # a grid that comes from a geometry and not from a power of two, the reference's default degree
        dict(name="step_mixed_odd", kind="step", steps=1, solver="pcg", mixed=True, precond="chebyshev", degree=5,
             **_grid(161, 93, 75, 1 / 93)),
        # the headline configuration
        dict(name="step_mixed_large", kind="step", steps=1, solver="pcg", mixed=True, precond="chebyshev", degree=4,
             **_grid(256, 128, 128, 1 / 128)),
        # the largest single case
        dict(name="step_mixed_xlarge", kind="step", steps=1, solver="pcg", mixed=True, precond="chebyshev", degree=4,
             **_grid(512, 256, 256, 1 / 256)),
        # the headline grid in the reference's arithmetic
        dict(name="step_fp64_large", kind="step", steps=1, solver="pcg", mixed=False, precond="chebyshev", degree=4,
             **_grid(256, 128, 128, 1 / 128)),
        # the headline grid with the lexicographic SOR solver, the reference's 200 sweeps
        dict(name="step_gs_large", kind="step", steps=1, solver="gs", mixed=False, precond="", degree=0,
             **_grid(256, 128, 128, 1 / 128)),
        # the stationary Jacobi solver (100 sweeps) on an ordinary grid whose spacing is no power of two
        dict(name="step_jacobi_mid", kind="step", steps=1, solver="jacobi", mixed=False, precond="", degree=0,
             **_grid(200, 100, 100, 1 / 100)),
        # the ensemble configuration: 64 ragged cases
        dict(name="ensemble_64", kind="ensemble", count=64, shapes=7, step=16, low=32, high=96, steps=2),
        # the gradient configuration over fewer steps
        dict(name="adjoint_mid", kind="adjoint", steps=10, every=5, **_grid(128, 64, 64, 1 / 64)),
        # a host loop that keeps its own step and calls each function
        dict(name="calls_mid", kind="calls", **_grid(128, 64, 64, 1 / 64)),
        # a symmetric system that the caller installs, IC(0)-PCG
        dict(name="pcg_ic_stored", kind="pcg", mixed=False, **_grid(96, 64, 64, 1 / 64)),
    ]


def _draw_grid(rng, lo, hi, longest=512):
    """A grid of lo to hi cells (spread over the logarithm), spacings as meshes have them."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ax, az = rng.uniform(1.0, 3.0), rng.uniform(0.6, 1.4)
    ny = (n / (ax * az)) ** (1 / 3)
    dims = [min(longest, max(12, int(round(v)))) for v in (ax * ny, ny, az * ny)]
    r = rng.random()
    if r < 0.4:  # sizes as the configurations have them
        dims = [min(longest, max(16, 16 * int(round(v / 16)))) for v in dims]
    h = 1.0 / dims[1] if r >= 0.3 else 0.5 ** int(round(math.log2(dims[1])))
    if 0.4 <= r < 0.6:  # other spacings along x and z
        return _grid(*dims, h * rng.uniform(0.8, 1.25), h, h * rng.uniform(0.8, 1.25))
    return _grid(*dims, h)


def draw(rng):
    r = rng.random()
    if r < 0.35:
        pc = rng.choice(["chebyshev", "chebyshev", "chebyshev", "jacobi"])
        g = _draw_grid(rng, 1 << 14, (1 << 23) if pc == "chebyshev" else (1 << 21))
        small = g["nx"] * g["ny"] * g["nz"] < (1 << 18)
        return dict(kind="step", steps=rng.randint(1, 4) if small else 1, solver="pcg", mixed=True, precond=pc,
                    degree=rng.choice([3, 4, 4, 5, 6]) if pc == "chebyshev" else 0, **g)
    if r < 0.50:
        pc = rng.choice(["chebyshev", "jacobi"])
        return dict(kind="step", steps=1, solver="pcg", mixed=False, precond=pc,
                    degree=rng.choice([3, 4, 5]) if pc == "chebyshev" else 0, **_draw_grid(rng, 1 << 13, 1 << 20))
    if r < 0.62:
        return dict(kind="step", steps=1, solver="gs", mixed=False, precond="", degree=0,
                    **_draw_grid(rng, 1 << 13, 1 << 22, 256))
    if r < 0.72:
        return dict(kind="step", steps=1, solver="jacobi", mixed=False, precond="", degree=0,
                    **_draw_grid(rng, 1 << 13, 1 << 23))
    if r < 0.80:
        return dict(kind="ensemble", count=rng.randint(4, 32), shapes=rng.randrange(1 << 20), step=rng.choice([1, 16]),
                    low=32, high=96, steps=rng.randint(1, 3))
    if r < 0.86:
        every = rng.randint(2, 4)
        return dict(kind="adjoint", steps=every * 2 + rng.randint(0, 1), every=every, **_draw_grid(rng, 1 << 14, 1 << 18))
    if r < 0.93:
        return dict(kind="calls", **_draw_grid(rng, 1 << 14, 1 << 23))
    return dict(kind="pcg", mixed=rng.random() < 0.4, **_draw_grid(rng, 1 << 13, 1 << 19))


# ---- inputs ---------------------------------------------------------------------
def _shape(c):
    return c["nx"], c["ny"], c["nz"]


def _spacing(c):
    return c["dx"], c["dy"], c["dz"]


def _box(shape):
    """The configurations' obstacle: a cube of a quarter of the cross-section, a quarter down the channel."""
    nx, ny, nz = shape
    return nx // 4, nx // 4 + max(2, ny // 4), 3 * ny // 8, 3 * ny // 8 + max(2, ny // 4), 3 * nz // 8, 3 * nz // 8 + max(2, nz // 4)


def _mask(shape, box):
    s = torch.zeros(shape, dtype=torch.bool, device="cuda")
    s[box[0]:box[1], box[2]:box[3], box[4]:box[5]] = True
    return s


def _velocity_bcs(vel, solid, inlet=None):
    """No slip at the walls, inflow, outflow, then the obstacle."""
    inner = torch.zeros_like(solid)
    inner[1:-1, 1:-1, 1:-1] = solid[1:-1, 1:-1, 1:-1]
    out = []
    for q, a in enumerate(vel):
        b = a.clone()
        flow = (torch.ones_like(a[0]) if inlet is None else inlet) if q == 0 else torch.zeros_like(a[0])
        b[0] = torch.where(solid[0], a[0], flow)
        b[-1] = a[-2]
        b[:, 0] = 0
        b[:, -1] = 0
        b[:, :, 0] = 0
        b[:, :, -1] = 0
        out.append(torch.where(inner, torch.zeros_like(b), b))
    return out


def _noise(shape, gen, amp):
    r = lambda: (2 * torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen) - 1) * amp  # noqa: E731
    return [1 + r(), r(), r()]


def _fields(shape, solid, seed, amp=NOISE):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    vel = _velocity_bcs(_noise(shape, gen, amp), solid)
    z = torch.zeros(shape, dtype=torch.float64, device="cuda")
    return dict(u=vel[0], v=vel[1], w=vel[2], p=z, nu_t=z)


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _to_host(fields):
    out = {}
    for k, a in fields.items():
        out[k] = _pinned(tuple(a.shape))
        out[k].copy_(a)
    return out


def _ptrs(d):
    return {k: a.data_ptr() for k, a in d.items()}


def _matrix_and_mask(ctx, solid, lam=True):
    """The matrix before the obstacle, then the mask."""
    n = solid.numel()
    ctx.upload_mask(np.zeros(n, np.uint8))
    ctx.build_stencil()
    lmax = ctx.lambda_max(20) if lam else 0.0
    ctx.upload_mask(solid.to(torch.uint8).cpu().numpy().reshape(-1))
    return lmax


def _step_params(c, lmax, cs=CS):
    mixed = c.get("mixed", True)
    pcg = G.pcg_opts(precond=PRECOND.get(c.get("precond"), G.PC_CHEBYSHEV), max_iter=20000, lambda_min=3 * math.pi ** 2,
                     lambda_max=lmax, degree=c.get("degree") or 4, precision=G.MIXED if mixed else G.FP64,
                     inner_rtol=1e-4, inner_max_iter=5000, max_outer=40)
    solver = SOLVER[c.get("solver", "pcg")]
    return G.step_params(nu=NU, rho=RHO, cs=cs, cfl_conv=CFL_CONV, cfl_visc=CFL_VISC, dt_max=DT_MAX, solver=solver,
                         rel_tol=MIXED_TOL if mixed else FP64_TOL, pcg=pcg,
                         stat_max_iter=100 if solver == G.SOLVER_JACOBI else 200, stat_tol=1e-6, omega=1.7)


def _ensemble(c):
    """The ensemble's shapes, obstacles and constants: of the case, not of the fields' seed."""
    rng = np.random.default_rng(c["shapes"])
    dims = np.arange(c["low"], c["high"] + 1, c["step"])
    out = []
    for _ in range(c["count"]):
        shape = tuple(int(rng.choice(dims)) for _ in range(3))
        side = min(shape) // 4
        pos = [int(rng.integers(1, n - side - 1)) for n in shape]
        out.append((shape, sum(((a, a + side) for a in pos), ()), float(rng.uniform(0.1, 0.2))))
    return out


def _probe(shape):
    nx, ny, nz = shape
    return 3 * nx // 4, nx - max(1, nx // 16), ny // 4, 3 * ny // 4, nz // 4, 3 * nz // 4


def _inlet(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) + 77)
    return 1 + 0.02 * (torch.rand((c["ny"], c["nz"]), dtype=torch.float64, device="cuda", generator=gen) - 0.5)


def _dirichlet_diagonals(c):
    """7-point -div grad with zero values outside the grid, as seven diagonals."""
    shape, inv = _shape(c), [1 / h ** 2 for h in _spacing(c)]
    n, d = shape, {"c": np.full(shape, 2 * sum(inv))}
    for axis, (lo, hi) in enumerate((("w", "e"), ("s", "n"), ("b", "t"))):
        for key, at in ((lo, 0), (hi, n[axis] - 1)):
            a = np.full(shape, -inv[axis])
            a[tuple(at if q == axis else slice(None) for q in range(3))] = 0.0
            d[key] = a
    return {k: a.reshape(-1) for k, a in d.items()}


def _pressure_guess(shape, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) + 5)
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)


def prepare(case, seed):
    c = case
    if c["kind"] == "ensemble":
        specs = _ensemble(c)
        ens = G.Ensemble([G.Mesh(*shape, 1 / 32, 1 / 32, 1 / 32) for shape, _, _ in specs])
        total = sum(math.prod(s) for s, _, _ in specs)
        out = {k: _pinned((total,)) for k in ("u", "v", "w", "p", "nu_t")}
        prm, ups, downs, at = [], [], [], 0
        for q, (shape, box, cs) in enumerate(specs):
            solid = _mask(shape, box)
            ctx, n = ens.cases[q], math.prod(shape)
            prm.append(_step_params(c, _matrix_and_mask(ctx, solid), cs))
            ups.append(_to_host(_fields(shape, solid, seed * 1000 + q, 0.02)))
            downs.append({k: a[at:at + n].data_ptr() for k, a in out.items()})
            at += n
        return dict(kind="ensemble", ens=ens, prm=prm, keep=ups, up=[_ptrs(u) for u in ups], down=downs, out=out,
                    steps=c["steps"])
    shape = _shape(c)
    ctx = G.Context(G.Mesh(*shape, *_spacing(c)))
    solid = _mask(shape, _box(shape))
    if c["kind"] == "pcg":
        ctx.set_stencil(_dirichlet_diagonals(c))
        ctx.build_ic()
        b = _to_host(dict(b=_pressure_guess(shape, seed), p=torch.zeros(shape, dtype=torch.float64, device="cuda")))
        tol = 1e-10 * float(torch.linalg.vector_norm(b["b"]))
        opts = G.pcg_opts(precond=G.PC_IC, max_iter=2000, tol=tol, precision=G.MIXED if c["mixed"] else G.FP64,
                          inner_max_iter=2000, max_outer=40)
        out = dict(p=_pinned(shape))
        return dict(kind="pcg", ctx=ctx, opts=opts, keep=b, up=_ptrs(b), out=out, down=_ptrs(out))
    lmax = _matrix_and_mask(ctx, solid, c["kind"] != "calls")
    f = _fields(shape, solid, seed)
    if c["kind"] == "adjoint":
        ctx.set_inlet(_inlet(c, seed).cpu().numpy())
        prm = _step_params(c, lmax)
        prm.dt_fixed = DT_MAX
        h = _to_host(f)
        return dict(kind="adjoint", ctx=ctx, prm=prm, keep=h, up=_ptrs(h), steps=c["steps"], every=c["every"],
                    box=_probe(shape))
    if c["kind"] == "calls":
        f["p"] = _pressure_guess(shape, seed)
        h = _to_host(f)
        out = {k: _pinned(shape) for k in ("u", "v", "w", "p", "nu_t", "b")}
        return dict(kind="calls", ctx=ctx, keep=h, up=_ptrs(h), out=out, down=_ptrs(out))
    h = _to_host(f)
    out = {k: _pinned(shape) for k in ("u", "v", "w", "p", "nu_t")}
    return dict(kind="step", ctx=ctx, prm=_step_params(c, lmax), keep=h, up=_ptrs(h), out=out, down=_ptrs(out),
                steps=c["steps"])


def run(state):
    s = state
    if s["kind"] == "step":
        if s["steps"] == 1:
            s["ctx"].step_io(s["prm"], s["up"], s["down"])
            return s["out"]
        s["ctx"].upload_many_ptr(s["up"])
        for _ in range(s["steps"]):
            s["ctx"].step(s["prm"])
        s["ctx"].download_many_ptr(s["down"])
        return s["out"]
    if s["kind"] == "ensemble":
        for ctx, up in zip(s["ens"].cases, s["up"]):
            ctx.upload_many_ptr(up)
        for _ in range(s["steps"]):
            s["ens"].step(s["prm"])
        for ctx, down in zip(s["ens"].cases, s["down"]):
            ctx.download_many_ptr(down)
        return s["out"]
    ctx = s["ctx"]
    ctx.upload_many_ptr(s["up"])
    if s["kind"] == "adjoint":
        j = ctx.adjoint_forward(s["prm"], s["steps"], s["every"], s["box"], MIXED_TOL)
        grad, gcs = ctx.adjoint_backward()
        return dict(j=j, grad=grad, grad_cs=gcs)
    if s["kind"] == "pcg":
        ctx.pcg(s["opts"])
        ctx.download_many_ptr(s["down"])
        return s["out"]
    dt = ctx.adaptive_dt(NU, CFL_CONV, CFL_VISC, DT_MAX)
    ctx.sgs_nut(CS)
    ctx.momentum(dt, NU)
    ctx.velocity_bcs()
    ctx.divergence(dt, RHO)
    ctx.build_b()
    ctx.pressure_bcs()
    ctx.correct_velocity(dt, RHO)
    ctx.velocity_bcs()
    energy = ctx.dot("u", "u")
    ctx.download_many_ptr(s["down"])
    return dict(s["out"], dt=dt, energy=energy)


def work(case):
    """Fields that come in and go out, each once; the stationary solvers' sweeps are asked for by number."""
    c = case
    if c["kind"] == "ensemble":
        n = sum(math.prod(s) for s, _, _ in _ensemble(c))
        return {"bytes": 81.0 * n, "flops": 120.0 * n * c["steps"]}
    n = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "pcg":
        return {"bytes": 80.0 * n, "flops": 40.0 * n}
    if c["kind"] == "adjoint":
        return {"bytes": 40.0 * n, "flops": 500.0 * n * c["steps"]}
    if c["kind"] == "calls":
        return {"bytes": 89.0 * n, "flops": 120.0 * n}
    sweeps = {"gs": 200, "jacobi": 100}.get(c["solver"], 0)
    return {"bytes": 81.0 * n, "flops": (120.0 * c["steps"] + 14.0 * sweeps) * n}


# ---- the same in 64 bits, by plain torch -----------------------------------------
def _d(a, axis):
    """a[+1] - a[-1] on the interior."""
    s = [slice(1, -1)] * 3
    hi, lo = list(s), list(s)
    hi[axis], lo[axis] = slice(2, None), slice(None, -2)
    return a[tuple(hi)] - a[tuple(lo)]


def _lap(a, h):
    s = [slice(1, -1)] * 3
    c, out = a[1:-1, 1:-1, 1:-1], 0
    for axis in range(3):
        hi, lo = list(s), list(s)
        hi[axis], lo[axis] = slice(2, None), slice(None, -2)
        out = out + (a[tuple(hi)] - 2 * c + a[tuple(lo)]) / h[axis] ** 2
    return out


def _nu_t(vel, solid, h, cs):
    g = [[_d(a, x) / (2 * h[x]) for x in range(3)] for a in vel]
    diag = g[0][0] ** 2 + g[1][1] ** 2 + g[2][2] ** 2
    off = ((g[0][1] + g[1][0]) / 2) ** 2 + ((g[0][2] + g[2][0]) / 2) ** 2 + ((g[1][2] + g[2][1]) / 2) ** 2
    sq = 2 * diag + 4 * off
    some = sq > 0
    s = torch.where(some, torch.sqrt(torch.where(some, sq, torch.ones_like(sq))), torch.zeros_like(sq))
    raw = (cs * (h[0] * h[1] * h[2]) ** (1 / 3)) ** 2 * s
    out = torch.zeros_like(vel[0])
    out[1:-1, 1:-1, 1:-1] = torch.where(solid[1:-1, 1:-1, 1:-1], torch.zeros_like(raw), raw)
    out[-1, 1:-1, 1:-1] = raw[-1]
    return out


def _momentum(vel, nu_t, h, dt):
    out = []
    core = [a[1:-1, 1:-1, 1:-1] for a in vel]
    for a in vel:
        adv = sum(core[x] * _d(a, x) / (2 * h[x]) for x in range(3))
        b = a.clone()
        b[1:-1, 1:-1, 1:-1] = a[1:-1, 1:-1, 1:-1] + dt * ((NU + nu_t[1:-1, 1:-1, 1:-1]) * _lap(a, h) - adv)
        out.append(b)
    return out


def _rhs(vel, solid, h, dt):
    """b = -(rho/dt) div u, one-sided at the boundary, zero in the obstacle and at the outlet."""
    div = 0
    for x, a in enumerate(vel):
        a = a.movedim(x, 0)
        d = torch.cat([(a[1:2] - a[:1]) / h[x], (a[2:] - a[:-2]) / (2 * h[x]), (a[-1:] - a[-2:-1]) / h[x]])
        div = div + d.movedim(0, x)
    off = solid.clone()
    off[-1] = True
    return torch.where(off, torch.zeros_like(div), -(RHO / dt) * div)


def _axis(n, h, left, right):
    """Eigenvectors (and their inverse) and eigenvalues of -d2/dx2 on n points; a mirrored end doubles its neighbour."""
    w = torch.ones(n, dtype=torch.float64, device="cuda")
    w[0] = 0.5 if left else 1.0
    w[-1] = 0.5 if right else w[-1]
    t = 2 * torch.eye(n, dtype=torch.float64, device="cuda")
    off = torch.ones(n - 1, dtype=torch.float64, device="cuda")
    off[0] = math.sqrt(2.0) if left else 1.0
    off[-1] = off[-1] * (math.sqrt(2.0) if right else 1.0)
    t = t - torch.diag(off, 1) - torch.diag(off, -1)
    lam, q = torch.linalg.eigh(t / h ** 2)
    return q / w.sqrt()[:, None], q.T * w.sqrt(), lam


def _poisson(h, shape, mirrored=True):
    """The solver of the pressure system by its eigenvectors; mirrored=False: zero values all around."""
    ends = ((True, False), (True, True), (True, True)) if mirrored else ((False, False),) * 3
    n = (shape[0] - 1 if mirrored else shape[0], shape[1], shape[2])
    ax = [_axis(n[q], h[q], *ends[q]) for q in range(3)]
    lam = ax[0][2][:, None, None] + ax[1][2][None, :, None] + ax[2][2]

    def along(m, a, x):
        return torch.tensordot(m, a, dims=([1], [x])).movedim(0, x)

    def solve(b):
        a = b[:-1] if mirrored else b
        for x in range(3):
            a = along(ax[x][1], a, x)
        a = a / lam
        for x in range(3):
            a = along(ax[x][0], a, x)
        return torch.cat([a, torch.zeros_like(b[:1])]) if mirrored else a

    return solve


def _pressure_bcs(p, solid):
    core = p[1:-1, 1:-1, 1:-1]
    p = torch.nn.functional.pad(core[None, None], (1,) * 6, mode="replicate")[0, 0].clone()
    p[-1] = 0
    out = p.clone()
    s = solid[1:-1, 1:-1, 1:-1]
    for axis, step in ((2, -1), (2, 1), (1, -1), (1, 1), (0, -1), (0, 1)):  # the first fluid neighbour wins
        at = [slice(1, -1)] * 3
        at[axis] = slice(2, None) if step > 0 else slice(None, -2)
        at = tuple(at)
        c = out[1:-1, 1:-1, 1:-1]
        out[1:-1, 1:-1, 1:-1] = torch.where(s & ~solid[at], p[at], c)
    return out


def _interior_rhs(vel, h, dt):
    r = torch.zeros_like(vel[0])
    r[1:-1, 1:-1, 1:-1] = RHO / dt * sum(_d(a, x) / (2 * h[x]) for x, a in enumerate(vel))
    return r


def _jacobi(p, vel, solid, h, dt):
    rhs, den = _interior_rhs(vel, h, dt)[1:-1, 1:-1, 1:-1], 2 * sum(1 / x ** 2 for x in h)
    for _ in range(100):
        c = p[1:-1, 1:-1, 1:-1]
        new = (_lap(p, h) + den * c - rhs) / den
        far = (new - c).abs().max()
        p = p.clone()
        p[1:-1, 1:-1, 1:-1] = new
        p = _pressure_bcs(p, solid)
        if float(far) < 1e-6:
            break
    return p


def _gs(p, vel, solid, h, dt, omega=1.7):
    """SOR in the lexicographic order: one plane i + j + k = const at a time."""
    shape = p.shape
    si, sj = shape[1] * shape[2], shape[2]
    i, j, k = torch.meshgrid(*[torch.arange(1, n - 1, device="cuda") for n in shape], indexing="ij")
    plane, at = (i + j + k).reshape(-1).sort(stable=True)
    ids = (i * si + j * sj + k).reshape(-1)[at]
    planes = ids.split(torch.unique_consecutive(plane, return_counts=True)[1].tolist())
    rhs, a = _interior_rhs(vel, h, dt).reshape(-1), p.reshape(-1).clone()
    coef = 1 / (2 * sum(1 / x ** 2 for x in h))

    def sweep():
        for q in planes:
            new = sum((a[q + s] + a[q - s]) / x ** 2 for s, x in zip((si, sj, 1), h)) - rhs[q]
            a[q] = (1 - omega) * a[q] + omega * coef * new

    start = a.clone()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        sweep()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sweep()
    a.copy_(start)
    for _ in range(200):
        old = a.clone()
        graph.replay()
        far = (a - old).abs().max()
        a.copy_(_pressure_bcs(a.reshape(shape), solid).reshape(-1))
        if float(far) < 1e-6:
            break
    return a.reshape(shape)


def _dt(vel, h):
    u = math.sqrt(float(sum(a ** 2 for a in vel).max()))
    return min(CFL_CONV * min(h) / u, CFL_VISC * min(h) ** 2 / NU, DT_MAX)


def _advance(vel, p, solid, h, dt, cs, solver, solve, inlet=None):
    nu_t = _nu_t(vel, solid, h, cs)
    new = _velocity_bcs(_momentum(vel, nu_t, h, dt), solid, inlet)
    if solver == "pcg":
        p = solve(_rhs(vel, solid, h, dt))
    else:
        p = (_gs if solver == "gs" else _jacobi)(p, new, solid, h, dt)
    out = []
    for x, a in enumerate(new):
        b = a.clone()
        b[1:-1, 1:-1, 1:-1] = a[1:-1, 1:-1, 1:-1] - dt / RHO * _d(p, x) / (2 * h[x])
        out.append(b)
    return _velocity_bcs(out, solid, inlet), p, nu_t


def _steps(shape, h, solid, f, steps, solver, cs):
    solve = _poisson(h, shape) if solver == "pcg" else None
    vel, p, nu_t = [f["u"], f["v"], f["w"]], f["p"], f["nu_t"]
    for n in range(steps):
        # nu_t of the step before is far below the viscous limit of dt on these grids
        vel, p, nu_t = _advance(vel, p, solid, h, _dt(vel, h), cs, solver, solve)
    return dict(u=vel[0], v=vel[1], w=vel[2], p=p, nu_t=nu_t)


def exact(case, seed):
    c = case
    if c["kind"] == "ensemble":
        got = []
        for q, (shape, box, cs) in enumerate(_ensemble(c)):
            solid = _mask(shape, box)
            f = _fields(shape, solid, seed * 1000 + q, 0.02)
            got.append(_steps(shape, (1 / 32,) * 3, solid, f, c["steps"], "pcg", cs))
        return {k: torch.cat([g[k].reshape(-1) for g in got]) for k in got[0]}
    shape, h = _shape(c), _spacing(c)
    if c["kind"] == "pcg":
        return dict(p=_poisson(h, shape, False)(_pressure_guess(shape, seed)))
    solid = _mask(shape, _box(shape))
    f = _fields(shape, solid, seed)
    vel = [f["u"], f["v"], f["w"]]
    if c["kind"] == "calls":
        dt = _dt(vel, h)
        p = _pressure_bcs(_pressure_guess(shape, seed), solid)
        nu_t = _nu_t(vel, solid, h, CS)
        new = _velocity_bcs(_momentum(vel, nu_t, h, dt), solid)
        for x, a in enumerate(new):
            a[1:-1, 1:-1, 1:-1] -= dt / RHO * _d(p, x) / (2 * h[x])
        new = _velocity_bcs(new, solid)
        return dict(u=new[0], v=new[1], w=new[2], p=p, nu_t=nu_t, b=_rhs(vel, solid, h, dt), dt=dt,
                    energy=float((new[0] ** 2).sum()))
    if c["kind"] == "adjoint":
        solve = _poisson(h, shape)
        inlet = _inlet(c, seed).requires_grad_()
        cs = torch.tensor(CS, dtype=torch.float64, device="cuda", requires_grad=True)
        b = _probe(shape)
        vel, p, j = _velocity_bcs(vel, solid, inlet), f["p"], 0
        for _ in range(c["steps"]):
            vel, p, _ = _advance(vel, p, solid, h, DT_MAX, cs, "pcg", solve, inlet)
            j = j + sum((a[b[0]:b[1], b[2]:b[3], b[4]:b[5]] ** 2).sum() for a in vel) / 2 / c["steps"]
        j.backward()
        return dict(j=float(j), grad=inlet.grad.reshape(-1), grad_cs=float(cs.grad))
    return _steps(shape, h, solid, f, c["steps"], c["solver"], CS)
