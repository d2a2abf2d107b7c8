"""The work whose speed is tracked: what programs built on this framework have it do, through its
public entry points, over the range of sizes, solvers and types they use.

Kinds of case (a case's ``kind``):

* ``poisson``: -Lap u = f to 1e-10 by CG with the vertex multigrid V(2,2)-cycle as preconditioner,
  the repository's headline solve (4095 x 4095 interior points).  ``cycle`` is the precision of the
  V-cycle inside the FP64 solver.  Small grids stand for solves inside a time loop, where launches
  and latency count; the others for one large stationary solve.
* ``convdiff``: convection-dominated convection-diffusion with the stream-function velocities of the
  benchmark, flexible GMRES(30) or BiCGSTAB with the convection-diffusion V-cycle.
* ``batch``: many such problems of uneven size solved together (a parameter study).
* ``explicit``: the explicit diffusion stepper (Euler, Heun, Runge-Kutta 4), some steps of it.
* ``implicit``: Crank-Nicolson steps solved by CG with the reference-hierarchy multigrid, Jacobi or
  Chebyshev smoothing: what a program written for the reference's steppers runs.
* ``krylov``: an implicit diffusion system without a preconditioner, on a grid no hierarchy fits.
* ``residual``: the residual of such a system and its norm by the field operations, in either type.
* ``training``: loss and gradient of the learned smoother over a set of samples.
"""
import math

import numpy as np
import torch

from fluxion_b200 import (BiCgStabSolver, Boundaries, CgSolver, ConvDiffMultigrid, ConvDiffOperator, Device, DType,
                          FgmresSolver, Field, GmresSolver, Grid, Multigrid, PipelinedCgSolver, SmootherKind, Stencil)
from fluxion_b200.batch import BatchSolver
from fluxion_b200.learned import LearnedSmoother, SmootherSamples
from fluxion_b200.steppers import CrankNicolsonSolver, DiffusionSolver, TimeScheme


def listed():
    return [
        # the headline solve: one large stationary Poisson problem, everything in FP64
        {"name": "poisson_4095_f64", "kind": "poisson", "rows": 4097, "cols": 4097, "cycle": "f64"},
        # an ordinary solve with the FP32 cycle, on a rectangle
        {"name": "poisson_1023x1279_f32", "kind": "poisson", "rows": 1025, "cols": 1281, "cycle": "f32"},
        # the smallest solve: a pressure equation on a coarse grid, launch latency
        {"name": "poisson_63_f64", "kind": "poisson", "rows": 65, "cols": 65, "cycle": "f64"},
        # the convection-dominated configuration of the benchmark
        {"name": "convdiff_fgmres_4095", "kind": "convdiff", "side": 4097, "nu": 1e-3, "solver": "fgmres",
         "cycle": "f64"},
        # an ordinary convection-diffusion solve
        {"name": "convdiff_bicgstab_1023", "kind": "convdiff", "side": 1025, "nu": 1e-2, "solver": "bicgstab",
         "cycle": "f64"},
        # a parameter study: 96 problems of 63 x 63 to 1023 x 1023, the tuned cycle precision
        {"name": "batch_96_f32", "kind": "batch", "count": 96, "kmin": 6, "kmax": 10, "cycle": "f32"},
        # explicit time stepping on an odd rectangle
        {"name": "explicit_rk4_1537x2050", "kind": "explicit", "rows": 1537, "cols": 2050, "scheme": "Rk4",
         "steps": 10, "graph": False},
        # one implicit step with the reference's default multigrid (Jacobi smoothing)
        {"name": "implicit_jacobi_256", "kind": "implicit", "rows": 256, "cols": 256, "smoother": "Jacobi"},
        # the same with Chebyshev smoothing, on a larger rectangle
        {"name": "implicit_chebyshev_1024x768", "kind": "implicit", "rows": 1024, "cols": 768,
         "smoother": "Chebyshev"},
        # an unpreconditioned solve on a ragged grid
        {"name": "pipelined_cg_1021x1531", "kind": "krylov", "rows": 1021, "cols": 1531, "solver": "pipelined_cg"},
        # monitoring a large single-precision simulation
        {"name": "residual_f32_8191x6001", "kind": "residual", "rows": 8191, "cols": 6001, "dtype": "f32"},
        # one large batch of the learned smoother's training
        {"name": "training_2048", "kind": "training", "samples": 2048, "lam": 0.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _vertex_side(rng, kmin, kmax):
    """A grid side the vertex hierarchy coarsens down to its coarsest grid: m 2^k + 1."""
    return rng.choice([4, 5, 6, 7]) * 2 ** rng.randint(kmin, kmax) + 1


def draw(rng):
    kind = rng.choice(["poisson", "poisson", "convdiff", "convdiff", "batch", "explicit", "implicit", "implicit",
                       "krylov", "residual", "training"])
    if kind == "poisson":
        k = rng.randint(4, 9)
        return {"kind": kind, "rows": _vertex_side(rng, k, k), "cols": _vertex_side(rng, k, k),
                "cycle": rng.choice(["f64", "f32"])}
    if kind == "convdiff":
        return {"kind": kind, "side": _vertex_side(rng, 4, 8), "nu": rng.choice([1e-2, 1e-3]),
                "solver": rng.choice(["fgmres", "bicgstab"]), "cycle": rng.choice(["f64", "f32"])}
    if kind == "batch":
        kmax = rng.randint(7, 10)
        return {"kind": kind, "count": rng.randint(17, 96), "kmin": 6, "kmax": kmax, "cycle": rng.choice(["f64", "f32"])}
    if kind == "explicit":
        return {"kind": kind, "rows": _log_int(rng, 48, 3000), "cols": _log_int(rng, 48, 3000),
                "scheme": rng.choice(["Euler", "Rk2", "Rk4"]), "steps": rng.randint(4, 16),
                "graph": rng.random() < 0.5}
    if kind == "implicit":
        # sides m 2^k with m in 3 .. 5: the reference hierarchy halves them exactly
        jacobi = rng.random() < 0.5
        k = rng.randint(3, 5) if jacobi else rng.randint(4, 7)
        return {"kind": kind, "rows": rng.choice([3, 4, 5]) * 2 ** k, "cols": rng.choice([3, 4, 5]) * 2 ** k,
                "smoother": "Jacobi" if jacobi else "Chebyshev"}
    if kind == "krylov":
        return {"kind": kind, "rows": _log_int(rng, 64, 2000), "cols": _log_int(rng, 64, 2000),
                "solver": rng.choice(["cg", "pipelined_cg", "bicgstab", "gmres"])}
    if kind == "residual":
        return {"kind": kind, "rows": _log_int(rng, 100, 8000), "cols": _log_int(rng, 100, 8000),
                "dtype": rng.choice(["f32", "f64"])}
    return {"kind": kind, "samples": _log_int(rng, 128, 4096), "lam": rng.choice([0.0, 0.3])}


# ---------------------------------------------------------------- inputs

def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _interior(rows, cols, seed, dtype=torch.float64):
    """U[-1, 1] inside, zero on the boundary ring."""
    f = torch.zeros(rows, cols, dtype=dtype, device="cuda")
    f[1:-1, 1:-1] = torch.rand(rows - 2, cols - 2, dtype=dtype, device="cuda", generator=_rng(seed)) * 2 - 1
    return f


def _smooth(rows, cols, seed):
    """A sum of sines with a little noise, zero on the ring: a field in the course of a simulation."""
    r = np.random.default_rng(seed)
    y = torch.arange(rows, dtype=torch.float64, device="cuda")[:, None] * (math.pi / (rows - 1))
    x = torch.arange(cols, dtype=torch.float64, device="cuda")[None, :] * (math.pi / (cols - 1))
    u = 0.05 * _interior(rows, cols, seed)
    for _ in range(6):
        k, l = (int(v) for v in r.integers(1, 9, 2))
        u += float(r.normal()) * torch.sin(k * y) * torch.sin(l * x)
    u[0], u[-1], u[:, 0], u[:, -1] = 0, 0, 0, 0
    return u


def _velocity(side, seed):
    """The benchmark's velocities: psi = sum of 8 modes a sin(k pi x) sin(l pi y), max |v| = 1."""
    r = np.random.default_rng(seed)
    t = torch.arange(side, dtype=torch.float64, device="cuda") * (math.pi / (side - 1))
    x, y = t[None, :], t[:, None]
    vx = torch.zeros(side, side, dtype=torch.float64, device="cuda")
    vy = torch.zeros_like(vx)
    for _ in range(8):
        k, l = (int(v) for v in r.integers(1, 5, 2))
        a = float(r.normal())
        vx += (a * l * math.pi) * torch.sin(k * x) * torch.cos(l * y)
        vy -= (a * k * math.pi) * torch.cos(k * x) * torch.sin(l * y)
    m = torch.sqrt(vx * vx + vy * vy).max()
    return vx / m, vy / m


def _field(t, grid, dev):
    """A field over a tensor's memory."""
    d = DType.F64 if t.dtype == torch.float64 else DType.F32
    return Field(dev.backend().wrap(t.data_ptr(), t.numel(), d), grid, dev)


def _dtype(name):
    return DType.F64 if name == "f64" else DType.F32


def _spacing(case):
    return 1.0 / (max(case["rows"], case["cols"]) - 1)


def _batch_sides(case):
    r = np.random.default_rng(case["count"])  # the mix belongs to the study, its data to the seed
    return [2 ** int(k) + 1 for k in r.integers(case["kmin"], case["kmax"] + 1, case["count"])]


_NU_BATCH = 1e-2
_CN = {"alpha": 1.0, "dt": 0.1, "tol": 1e-8, "max_iter": 100}


def _krylov_coeff(h):
    return -25.0 * h * h  # half a step of 50 h^2


_TOL = {"cg": 1e-10, "pipelined_cg": 1e-10, "bicgstab": 1e-10, "gmres": 1e-8}


def prepare(case, seed):
    dev = Device.best()
    kind = case["kind"]
    s = {"kind": kind, "case": case, "dev": dev}
    if kind == "poisson":
        h = _spacing(case)
        g = Grid.new(case["rows"], case["cols"], h, h)
        s["ft"] = _interior(g.rows, g.cols, seed)
        s["xt"] = torch.zeros_like(s["ft"])
        torch.cuda.synchronize()
        s["f"], s["x"] = _field(s["ft"], g, dev), _field(s["xt"], g, dev)
        s["stencil"], s["bc"] = Stencil.poisson_neg_laplacian(h, h), Boundaries.zero_dirichlet()
        s["mg"] = Multigrid.vertex(g, s["bc"], dev, dtype=_dtype(case["cycle"]), op_stencil=s["stencil"])
        s["solver"] = CgSolver(g, dev, 1e-10 * float(s["ft"].norm()), 200)
    elif kind == "convdiff":
        n, h = case["side"], 1.0 / (case["side"] - 1)
        g = Grid.square(n, h)
        s["vxt"], s["vyt"] = _velocity(n, seed)
        s["ft"] = _interior(n, n, seed + 1)
        s["xt"] = torch.zeros_like(s["ft"])
        torch.cuda.synchronize()
        s["f"], s["x"] = _field(s["ft"], g, dev), _field(s["xt"], g, dev)
        s["op"] = ConvDiffOperator(g, _field(s["vxt"], g, dev), _field(s["vyt"], g, dev), -case["nu"], sigma=0.0)
        s["mg"] = ConvDiffMultigrid(s["op"], dtype=_dtype(case["cycle"]))
        tol = 1e-10 * float(s["ft"].norm())
        s["solver"] = FgmresSolver(g, dev, 30, tol, 2000) if case["solver"] == "fgmres" else BiCgStabSolver(
            g, dev, tol, 2000)
    elif kind == "batch":
        sides = _batch_sides(case)
        parts = [(_velocity(n, seed * 1000 + i), _interior(n, n, seed * 1000 + i)) for i, n in enumerate(sides)]
        s["vxt"] = torch.cat([v[0].reshape(-1) for v, _ in parts])
        s["vyt"] = torch.cat([v[1].reshape(-1) for v, _ in parts])
        s["ft"] = torch.cat([f.reshape(-1) for _, f in parts])
        s["xt"] = torch.zeros_like(s["ft"])
        torch.cuda.synchronize()
        be = dev.backend()
        for k in ("vx", "vy", "f", "x"):
            s[k] = be.wrap(s[k + "t"].data_ptr(), s[k + "t"].numel(), DType.F64)
        s["solver"] = BatchSolver(dev, sides, _NU_BATCH, s["vx"], s["vy"], cycle_dtype=_dtype(case["cycle"]))
    elif kind == "explicit":
        h = _spacing(case)
        g = Grid.new(case["rows"], case["cols"], h, h)
        s["u0t"] = _smooth(g.rows, g.cols, seed)
        s["ut"] = s["u0t"].clone()
        torch.cuda.synchronize()
        s["u0"], s["u"] = _field(s["u0t"], g, dev), _field(s["ut"], g, dev)
        s["solver"] = DiffusionSolver.build(g, 1.0, None, Boundaries.zero_dirichlet(), TimeScheme[case["scheme"]], dev)
        if case["graph"]:
            s["solver"].enable_graph()
    elif kind == "implicit":
        h = _spacing(case)
        g = Grid.new(case["rows"], case["cols"], h, h)
        s["u0t"] = _smooth(g.rows, g.cols, seed)
        s["ut"] = s["u0t"].clone()
        torch.cuda.synchronize()
        s["u0"], s["u"] = _field(s["u0t"], g, dev), _field(s["ut"], g, dev)
        s["solver"] = CrankNicolsonSolver.with_multigrid_smoother(
            g, _CN["alpha"], _CN["dt"], Boundaries.zero_dirichlet(), dev, _CN["tol"], _CN["max_iter"], 2, 2, 2.0 / 3.0,
            SmootherKind[case["smoother"]])
    elif kind == "krylov":
        h = _spacing(case)
        g = Grid.new(case["rows"], case["cols"], h, h)
        s["ft"] = _interior(g.rows, g.cols, seed)
        s["xt"] = torch.zeros_like(s["ft"])
        torch.cuda.synchronize()
        s["f"], s["x"] = _field(s["ft"], g, dev), _field(s["xt"], g, dev)
        s["stencil"], s["bc"], s["coeff"] = Stencil.laplacian_2d_5pt(h, h), Boundaries.zero_dirichlet(), _krylov_coeff(h)
        tol = _TOL[case["solver"]] * float(s["ft"].norm())
        s["solver"] = {"cg": lambda: CgSolver(g, dev, tol, 2000),
                       "pipelined_cg": lambda: PipelinedCgSolver(g, dev, tol, 2000),
                       "bicgstab": lambda: BiCgStabSolver(g, dev, tol, 2000),
                       "gmres": lambda: GmresSolver(g, dev, 30, tol, 2000)}[case["solver"]]()
    elif kind == "residual":
        h = _spacing(case)
        g = Grid.new(case["rows"], case["cols"], h, h)
        td = torch.float64 if case["dtype"] == "f64" else torch.float32
        s["bt"], s["xt"] = _interior(g.rows, g.cols, seed, td), _interior(g.rows, g.cols, seed + 1, td)
        s["rt"] = torch.zeros_like(s["bt"])
        torch.cuda.synchronize()
        s["b"], s["x"], s["r"] = (_field(s[k], g, dev) for k in ("bt", "xt", "rt"))
        s["stencil"], s["bc"], s["coeff"] = Stencil.laplacian_2d_5pt(h, h), Boundaries.zero_dirichlet(), _krylov_coeff(h)
    else:
        n = 513
        g = Grid.square(n, 1.0 / (n - 1))
        vxt, vyt = _velocity(n, seed)
        xt, et, bt = (_interior(n, n, seed + k) for k in (1, 2, 3))
        torch.cuda.synchronize()
        op = ConvDiffOperator(g, _field(vxt, g, dev), _field(vyt, g, dev), -1e-3, sigma=0.0)
        r = np.random.default_rng(seed)
        origins = 2 * r.integers(2, (n - 21) // 2, (case["samples"], 2))
        s["data"] = SmootherSamples(dev, case["samples"])
        s["data"].add_patches(op, _field(xt, g, dev), _field(et, g, dev), _field(bt, g, dev), 0.8, origins)
        dev.backend().synchronize()
        s["net"] = LearnedSmoother(dev, seed & 0xFFFF)
        p = s["net"].params
        # some way into the training: every layer carries weights and biases
        p[-145:-1] = r.normal(0.0, 0.1, 144)
        p[432:448], p[2752:2768] = r.normal(0.0, 0.05, 16), r.normal(0.0, 0.05, 16)
        s["net"].params = p
        s["index"] = r.permutation(case["samples"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "poisson":
        s["x"].fill(0.0)
        s["solver"].solve_preconditioned(s["x"], s["f"], 1.0, s["stencil"], s["bc"], s["mg"])
        return s["xt"]
    if kind == "convdiff":
        s["x"].fill(0.0)
        s["solver"].solve_op(s["x"], s["f"], s["op"], s["mg"])
        return s["xt"]
    if kind == "batch":
        s["dev"].backend().fill(s["x"], 0.0)
        s["solver"].bicgstab(s["x"], s["f"], 1e-10, 200)
        return s["xt"]
    if kind == "explicit":
        s["u"].copy_from(s["u0"])
        s["solver"].step_n(s["u"], s["case"]["steps"])
        return s["ut"]
    if kind == "implicit":
        s["u"].copy_from(s["u0"])
        s["solver"].step(s["u"])
        return s["ut"]
    if kind == "krylov":
        s["x"].fill(0.0)
        s["solver"].solve(s["x"], s["f"], s["coeff"], s["stencil"], s["bc"])
        return s["xt"]
    if kind == "residual":
        r, x = s["r"], s["x"]
        r.copy_from(s["b"])
        r.axpy(-1.0, x)
        r.stencil_axpy(-s["coeff"], x, s["stencil"], s["bc"])
        return {"r": s["rt"], "norm": r.norm_l2()}
    loss, grad = s["net"].loss_grad(s["data"], s["index"], True, s["case"]["lam"])
    return {"loss": loss, "grad": grad}


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    """Bytes of the algorithm's vectors and fields, each read and written once by each phase that
    an inner product or the cycle's structure separates from the next, times a typical iteration
    count; flops of the stencils and updates."""
    kind = case["kind"]
    if kind == "poisson":
        n = case["rows"] * case["cols"]
        # 9 iterations: direction 24, update 40, V-cycle (down 10, up 18 in FP64) with a third more for the coarse levels
        cyc = (28 if case["cycle"] == "f64" else 24) * 4 / 3
        return {"bytes": n * 9 * (24 + 40 + cyc), "flops": n * 9 * 100}
    if kind == "convdiff":
        n = case["side"] ** 2
        cyc = (34 + 42) * (1 if case["cycle"] == "f64" else 0.6) * 4 / 3
        if case["solver"] == "fgmres":
            its = 40 if case["nu"] < 5e-3 else 16
            # per iteration: cycle, w = A z (40), two reads of half of a 15-vector basis on average, norm and scaling
            return {"bytes": n * its * (cyc + 40 + 2 * 8 * 15 + 32), "flops": n * its * 300}
        its = 25 if case["nu"] < 5e-3 else 9
        return {"bytes": n * its * (216 + 2 * cyc), "flops": n * its * 500}
    if kind == "batch":
        ks = range(case["kmin"], case["kmax"] + 1)
        n = case["count"] * sum((2 ** k + 1) ** 2 for k in ks) / len(ks)
        cyc = (34 + 42) * (1 if case["cycle"] == "f64" else 0.6) * 4 / 3
        return {"bytes": n * 9 * (216 + 2 * cyc), "flops": n * 9 * 500}
    if kind == "explicit":
        n = case["rows"] * case["cols"]
        stages = {"Euler": 1, "Rk2": 2, "Rk4": 4}[case["scheme"]]
        # a step reads u and writes u; every further stage reads and writes one vector more
        return {"bytes": n * case["steps"] * (16 + 16 * (stages - 1)), "flops": n * case["steps"] * stages * 12}
    if kind == "implicit":
        n = case["rows"] * case["cols"]
        return {"bytes": n * 10 * (64 + 8 * 24 * 4 / 3), "flops": n * 10 * 150}
    if kind == "krylov":
        n = case["rows"] * case["cols"]
        per, its = {"cg": (64, 80), "pipelined_cg": (96, 80), "bicgstab": (168, 50),
                    "gmres": (24 + 2 * 8 * 15, 70)}[case["solver"]]
        return {"bytes": n * its * per, "flops": n * its * 30}
    if kind == "residual":
        n = case["rows"] * case["cols"] * (8 if case["dtype"] == "f64" else 4)
        # copy, axpy, stencil_axpy and the norm are calls of their own
        return {"bytes": n * (2 + 3 + 3 + 1), "flops": 2.5 * n}
    macs = 23 * 23 * 16 * 27 + 21 * 21 * 16 * 144 + 19 * 19 * 144  # one sample, forward
    return {"bytes": case["samples"] * (1875 * 2 + 512 * 4), "flops": case["samples"] * 2 * 3 * macs}


# ---------------------------------------------------------------- the same in plain FP64

def _dst_solve(f, shift, scale, h):
    """(shift - scale Lap_h) u = f inside with u = 0 on the ring, by sine transforms."""
    rows, cols = f.shape

    def dst(a):  # DST-I along the last axis by a real FFT of the odd extension
        z = torch.zeros(*a.shape[:-1], 1, dtype=a.dtype, device=a.device)
        return -torch.fft.rfft(torch.cat([z, a, z, -a.flip(-1)], -1)).imag[..., 1:-1]

    i = f[1:-1, 1:-1]
    t = dst(dst(i).T.contiguous()).T
    sr = torch.sin(torch.arange(1, rows - 1, dtype=torch.float64, device=f.device) * math.pi / (2 * (rows - 1))) ** 2
    sc = torch.sin(torch.arange(1, cols - 1, dtype=torch.float64, device=f.device) * math.pi / (2 * (cols - 1))) ** 2
    t = t / (shift + scale * (4.0 / (h * h)) * (sr[:, None] + sc[None, :]))
    u = torch.zeros_like(f)
    u[1:-1, 1:-1] = dst(dst(t.contiguous()).T.contiguous()).T / (4.0 * (rows - 1) * (cols - 1))
    return u


def _lap(u, h):
    out = torch.zeros_like(u)
    out[..., 1:-1, 1:-1] = (u[..., :-2, 1:-1] + u[..., 2:, 1:-1] + u[..., 1:-1, :-2] + u[..., 1:-1, 2:]
                            - 4 * u[..., 1:-1, 1:-1]) / (h * h)
    return out


class _ConvDiff:
    """-nu Lap u + v.grad u (first-order upwind) on square grids, leading dimension: problems."""

    def __init__(self, vx, vy, nu, h):
        self.nu, self.h, self.vx, self.vy = nu, h, vx, vy
        self.inv_diag = 1.0 / (4 * nu / (h * h) + (vx.abs() + vy.abs()) / h)[..., 1:-1, 1:-1]
        n = vx.shape[-1]
        self.coarse = _ConvDiff(vx[..., ::2, ::2], vy[..., ::2, ::2], nu, 2 * h) if n - 2 > 15 and n % 2 else None

    def apply(self, u):
        c, h = u[..., 1:-1, 1:-1], self.h
        vx, vy = self.vx[..., 1:-1, 1:-1], self.vy[..., 1:-1, 1:-1]
        ux = torch.where(vx >= 0, c - u[..., 1:-1, :-2], u[..., 1:-1, 2:] - c)
        uy = torch.where(vy >= 0, c - u[..., :-2, 1:-1], u[..., 2:, 1:-1] - c)
        out = torch.zeros_like(u)
        out[..., 1:-1, 1:-1] = -self.nu * _lap(u, h)[..., 1:-1, 1:-1] + (vx * ux + vy * uy) / h
        return out

    def smooth(self, x, b, n):
        for _ in range(n):
            x[..., 1:-1, 1:-1] += 0.8 * (b - self.apply(x))[..., 1:-1, 1:-1] * self.inv_diag

    def cycle(self, b):
        x = torch.zeros_like(b)
        if self.coarse is None:
            self.smooth(x, b, 200)
            return x
        self.smooth(x, b, 2)
        r = b - self.apply(x)
        rc = torch.zeros_like(self.coarse.vx)
        q = r[..., 1:-1, :]
        v = 0.25 * (r[..., :-2, :] + 2 * q + r[..., 2:, :])
        v = 0.25 * (v[..., :-2] + 2 * v[..., 1:-1] + v[..., 2:])
        rc[..., 1:-1, 1:-1] = v[..., 1::2, 1::2]
        e = self.coarse.cycle(rc)
        x[..., ::2, ::2] += e
        x[..., 1::2, ::2] += 0.5 * (e[..., :-1, :] + e[..., 1:, :])
        x[..., ::2, 1::2] += 0.5 * (e[..., :-1] + e[..., 1:])
        x[..., 1::2, 1::2] += 0.25 * (e[..., :-1, :-1] + e[..., 1:, :-1] + e[..., :-1, 1:] + e[..., 1:, 1:])
        self.smooth(x, b, 2)
        return x

    def solve(self, b, m=40, restarts=6):
        """Flexible GMRES with the cycle, until the residual no longer falls."""
        def dot(a, c):
            return (a * c).sum((-2, -1))

        x, best, last = torch.zeros_like(b), None, math.inf
        bn = dot(b, b).sqrt()
        for _ in range(restarts):
            r = b - self.apply(x)
            beta = dot(r, r).sqrt()
            rel = float((beta / bn).max())
            if rel < last:
                best, gain, last = x.clone(), last / rel, rel
            if rel < 1e-14 or gain < 2:
                break
            gain = 1.0
            V, Z = [r / beta[..., None, None]], []
            H = torch.zeros(b.shape[0], m + 1, m, dtype=torch.float64)
            for j in range(m):
                Z.append(self.cycle(V[j]))
                w = self.apply(Z[j])
                for _ in range(2):
                    for i, v in enumerate(V):
                        c = dot(w, v)
                        w -= c[..., None, None] * v
                        H[:, i, j] += c.cpu()
                nw = dot(w, w).sqrt()
                H[:, j + 1, j] = nw.cpu()
                V.append(w / nw.clamp_min(1e-300)[..., None, None])
            rhs = torch.zeros(b.shape[0], m + 1, 1, dtype=torch.float64)
            rhs[:, 0, 0] = beta.cpu()
            y = torch.linalg.lstsq(H, rhs, driver="gelsd").solution[..., 0].to(b.device)
            for j in range(m):
                x += y[:, j, None, None] * Z[j]
        return best


def _explicit_exact(case, u):
    h = _spacing(case)
    safety = {"Euler": 0.4, "Rk2": 0.8, "Rk4": 1.4}[case["scheme"]]
    dt = safety * h * h / 4.0
    for _ in range(case["steps"]):
        if case["scheme"] == "Euler":
            u = u + dt * _lap(u, h)
        elif case["scheme"] == "Rk2":
            v = u + dt * _lap(u, h)
            u = 0.5 * (u + v + dt * _lap(v, h))
        else:
            k1 = _lap(u, h)
            k2 = _lap(u + 0.5 * dt * k1, h)
            k3 = _lap(u + 0.5 * dt * k2, h)
            k4 = _lap(u + dt * k3, h)
            u = u + dt / 6.0 * (k1 + 2 * k2 + 2 * k3 + k4)
    return u


def exact(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        return _dst_solve(_interior(case["rows"], case["cols"], seed), 0.0, 1.0, _spacing(case))
    if kind == "convdiff":
        n = case["side"]
        vx, vy = _velocity(n, seed)
        return _ConvDiff(vx[None], vy[None], case["nu"], 1.0 / (n - 1)).solve(_interior(n, n, seed + 1)[None])[0]
    if kind == "batch":
        sides = _batch_sides(case)
        out = [None] * len(sides)
        for n in sorted(set(sides)):
            which = [i for i, m in enumerate(sides) if m == n]
            for at in range(0, len(which), 16):
                part = which[at:at + 16]
                v = [_velocity(n, seed * 1000 + i) for i in part]
                f = torch.stack([_interior(n, n, seed * 1000 + i) for i in part])
                u = _ConvDiff(torch.stack([a for a, _ in v]), torch.stack([b for _, b in v]), _NU_BATCH,
                              1.0 / (n - 1)).solve(f, m=24)
                for j, i in enumerate(part):
                    out[i] = u[j].reshape(-1)
        return torch.cat(out)
    if kind == "explicit":
        return _explicit_exact(case, _smooth(case["rows"], case["cols"], seed))
    if kind == "implicit":
        h, c = _spacing(case), 0.5 * _CN["dt"] * _CN["alpha"]
        u = _smooth(case["rows"], case["cols"], seed)
        return _dst_solve(u + c * _lap(u, h), 1.0, c, h)
    if kind == "krylov":
        h = _spacing(case)
        return _dst_solve(_interior(case["rows"], case["cols"], seed), 1.0, -_krylov_coeff(h), h)
    if kind == "residual":
        h = _spacing(case)
        td = torch.float64 if case["dtype"] == "f64" else torch.float32
        b = _interior(case["rows"], case["cols"], seed, td).double()
        x = _interior(case["rows"], case["cols"], seed + 1, td).double()
        r = b - x - _krylov_coeff(h) * _lap(x, h)
        return {"r": r, "norm": float(r.norm())}
    return None  # a BF16 network: its roundings are part of its definition
