"""Performance cases: the work that a user of the package has it do, by size and form.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges,
``prepare(case, seed)`` builds what a program holds before the call (the solver or
engine, the seeded state), ``run(state)`` is one pass through the public entry points,
``work(case)`` the bytes and operations a pass cannot do without, and
``exact(case, seed)`` the same outputs from plain float64 tensor arithmetic with a
spectral Poisson solve (grids without obstacles, uniform spacing).

Kinds of case:

* ``run``      ``TimeStepper.run`` for a few adaptive steps (the simulation loop)
* ``step``     ``ProjectionSolver.step`` (one RK3 step, new arrays)
* ``advance``  ``ProjectionSolver.advance`` (one RK3 step, replayed)
* ``batch``    ``BatchedSolver.step`` / ``ConcurrentBatch.step`` (one step of every problem)
* ``solve``    ``pressure_solver.solve`` (one Poisson solve from a zero start)
* ``stencil``  ``momentum_rhs`` and ``divergence`` of one velocity field
* ``adjoint``  ``objective_fn(...)`` and its ``backward()``
"""

from __future__ import annotations

import math

import numpy as np
import torch

from pycfd_b200.config import BCKind, BCSpec, SimulationConfig

F64 = torch.float64
TOL = 1e-10            # the package's own Poisson tolerance in its configurations
MG_ITERATIONS = 11     # MG-PCG iterations of one solve to 1e-10
LEVEL_SUM = 4.0 / 3.0  # cells of all multigrid levels over the fine level's (2 x 2 coarsening)


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest simulation: the 64 x 64 lid-driven cavity at Re 100 with
        # Jacobi-preconditioned CG, a short call of the simulation loop
        dict(name="cavity64_cg_run", kind="run", nx=64, ny=64, solver="cg", steps=4),
        # one step of an ordinary cavity with multigrid-preconditioned CG, the call of a
        # program that drives its own loop
        dict(name="cavity128_mgcg_step", kind="step", flow="cavity", nx=128, ny=128, precision="fp64"),
        # the 512 x 512 Taylor-Green vortex, the recorded FP64 step
        dict(name="vortex512_advance", kind="advance", flow="periodic", nx=512, ny=512, precision="fp64"),
        # the largest domain: flow past a cylinder on 2048 x 1024 cells (inflow,
        # convective outlet, slip walls), the recorded FP64 step
        dict(name="cylinder2048_advance", kind="advance", flow="cylinder", nx=2048, ny=1024,
             precision="fp64"),
        # the same flow on 512 x 256 cells in the mixed-precision form
        dict(name="cylinder512_mixed", kind="advance", flow="cylinder", nx=512, ny=256, precision="mixed"),
        # a channel past a cylinder on a stretched, odd-sized mesh with the Smagorinsky closure
        dict(name="stretched_les", kind="advance", flow="stretched", nx=301, ny=147, precision="fp64"),
        # the large batch: 256 cavities of 64^2 ... 256^2 in the mixed form, four
        # concurrent parts, the options the autotuner picks for it
        dict(name="batch256_mixed", kind="batch", sizes="64,96,128,192,256", count=256, precision="mixed",
             tuned=True, parts=4),
        # a small parameter study on odd grids, one engine with its default options
        dict(name="batch24_odd_mixed", kind="batch", sizes="50,77,101,130", count=24, precision="mixed",
             tuned=False, parts=1),
        # a middling batch in double precision, one engine
        dict(name="batch64_fp64", kind="batch", sizes="64,96,128,192", count=64, precision="fp64",
             tuned=False, parts=1),
        # one Poisson solve by Jacobi-preconditioned CG on a non-square grid
        dict(name="poisson_cg_200x150", kind="solve", solver="cg", nx=200, ny=150),
        # the momentum right-hand side and the divergence of a large field
        dict(name="stencil_1500x1100", kind="stencil", nx=1500, ny=1100, blend=0.2),
        # gradient of the cavity objective by the discrete adjoint (forward and backward sweep)
        dict(name="adjoint128", kind="adjoint", n=128, steps=3),
    ]


def _spread(rng, lo, hi):
    """A size between lo and hi, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("run", "step", "vortex", "cylinder", "stretched", "batch", "batch", "solve", "stencil",
                       "adjoint"))
    if kind == "run":
        return dict(kind="run", nx=_spread(rng, 24, 128), ny=_spread(rng, 24, 128), solver="cg",
                    steps=rng.randint(2, 6))
    if kind == "step":
        return dict(kind="step", flow="cavity", nx=_spread(rng, 40, 300), ny=_spread(rng, 40, 300),
                    precision="fp64")
    if kind == "vortex":
        return dict(kind="advance", flow="periodic", nx=_spread(rng, 64, 640), ny=_spread(rng, 64, 640),
                    precision=rng.choice(("fp64", "fp64", "mixed")))
    if kind == "cylinder":
        ny = _spread(rng, 96, 512)
        return dict(kind="advance", flow="cylinder", nx=2 * ny + rng.randint(-8, 8), ny=ny,
                    precision=rng.choice(("fp64", "mixed")))
    if kind == "stretched":
        ny = _spread(rng, 64, 200)
        return dict(kind="advance", flow="stretched", nx=2 * ny + rng.randint(-9, 9), ny=ny, precision="fp64")
    if kind == "batch":
        sizes = sorted(_spread(rng, 40, 256) for _ in range(rng.randint(2, 5)))
        count = _spread(rng, 8, 128)
        precision = rng.choice(("mixed", "mixed", "fp64"))
        parts = rng.choice((1, 1, 4))
        return dict(kind="batch", sizes=",".join(map(str, sizes)), count=count, precision=precision,
                    tuned=bool(parts > 1), parts=parts)
    if kind == "solve":
        return dict(kind="solve", solver=rng.choice(("cg", "mgcg")), nx=_spread(rng, 40, 320),
                    ny=_spread(rng, 40, 320))
    if kind == "stencil":
        return dict(kind="stencil", nx=_spread(rng, 100, 2000), ny=_spread(rng, 100, 2000),
                    blend=rng.choice((0.0, 0.2)))
    return dict(kind="adjoint", n=_spread(rng, 48, 160), steps=rng.randint(1, 4))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _walls(flow, lid=1.0):
    if flow == "periodic":
        return {w: BCSpec(BCKind.PERIODIC) for w in ("left", "right", "bottom", "top")}
    if flow in ("cylinder", "stretched"):
        side = BCKind.SYMMETRY if flow == "cylinder" else BCKind.NO_SLIP
        return {"left": BCSpec(BCKind.INLET, velocity=1.0,
                               profile="uniform" if flow == "cylinder" else "parabolic"),
                "right": BCSpec(BCKind.OUTLET), "bottom": BCSpec(side), "top": BCSpec(side)}
    walls = {w: BCSpec(BCKind.NO_SLIP) for w in ("left", "right", "bottom")}
    walls["top"] = BCSpec(BCKind.MOVING_WALL, velocity=lid)
    return walls


def _extent(case):
    """Domain size: cells are square on every flow but the stretched one."""
    nx, ny = case["nx"], case["ny"]
    if case.get("flow") == "periodic":
        return 2 * math.pi * nx / max(nx, ny), 2 * math.pi * ny / max(nx, ny)
    if case.get("flow") == "cylinder":
        return 2.0, 2.0 * ny / nx
    if case.get("flow") == "stretched":
        return 4.0, 1.0
    return nx / max(nx, ny), ny / max(nx, ny)


def _config(case):
    flow = case.get("flow", "cavity")
    lx, ly = _extent(case)
    kw = dict(nx=case["nx"], ny=case["ny"], lx=lx, ly=ly, re=400.0, dt=_dt(case), t_end=1e9, adaptive_dt=False,
              pressure_solver=case.get("solver", "mgcg"), poisson_tol=TOL, boundary_config=_walls(flow))
    if flow == "cylinder":
        kw.update(re=100.0, l_ref=0.1)
    if flow == "stretched":
        kw.update(re=2000.0, l_ref=0.2, stretch_x=1.002, stretch_y=1.01, cluster_y="walls", use_les=True)
    if case["kind"] == "run":
        kw.update(re=100.0, dt=1.0, adaptive_dt=True, cfl_max=0.5)
    return SimulationConfig(**kw)


def _dt(case):
    """A time step at CFL 0.3 of a unit velocity (the smallest cell of the stretched mesh)."""
    lx, ly = _extent(case)
    h = min(lx / case["nx"], ly / case["ny"])
    return 0.3 * h * (0.2 if case.get("flow") == "stretched" else 1.0)


def _modes(seed, k, periodic):
    """Wave numbers, phases and amplitudes of a seeded stream function."""
    rng = np.random.default_rng([int(seed), int(k)])
    m = rng.integers(1, 5, (6, 2))
    a = rng.standard_normal(6) / np.hypot(m[:, 0], m[:, 1])
    return m, a, rng.uniform(0, 2 * np.pi, (6, 2)) if periodic else np.zeros((6, 2))


def _velocity(nx, ny, lx, ly, seed, k=0, periodic=False, device="cpu"):
    """Divergence-free face velocities (nx+1, ny), (nx, ny+1) of a seeded stream function
    (zero on the walls of a closed box), about 0.3 in size."""
    m, a, ph = _modes(seed, k, periodic)
    x = torch.arange(nx + 1, dtype=F64, device=device) / nx
    y = torch.arange(ny + 1, dtype=F64, device=device) / ny
    c = (2 if periodic else 1) * math.pi
    psi = sum(float(a[q]) * torch.sin(c * int(m[q, 0]) * x + float(ph[q, 0]))[:, None]
              * torch.sin(c * int(m[q, 1]) * y + float(ph[q, 1]))[None, :] for q in range(len(a)))
    psi = 0.3 * max(lx, ly) / (2 * c) * psi
    return (psi[:, 1:] - psi[:, :-1]) * (ny / ly), -(psi[1:] - psi[:-1]) * (nx / lx)


def _single_init(case, seed, device):
    nx, ny = case["nx"], case["ny"]
    lx, ly = _extent(case)
    flow = case.get("flow", "cavity")
    u, v = _velocity(nx, ny, lx, ly, seed, 0, flow == "periodic", device)
    if flow == "cylinder":
        return 1.0 + 0.05 * u, 0.05 * v
    if flow == "stretched":
        return 0.5 + 0.05 * u, 0.05 * v
    return u, v


def _batch_problems(case, seed):
    """(n, Re, lid) of every cavity: sizes in turn, Re log-uniform 100 ... 2000, lid 0.5 ... 1.5."""
    sizes = [int(s) for s in case["sizes"].split(",")]
    rng = np.random.default_rng([int(seed), 77])
    n = [sizes[k % len(sizes)] for k in range(case["count"])]
    re = np.exp(rng.uniform(np.log(100.0), np.log(2000.0), len(n)))
    lid = rng.uniform(0.5, 1.5, len(n))
    return n, re, lid


def _fields(seed, shape_u, shape_v, device):
    """Random ghosted velocities of the stencil case: a smooth flow with noise on it."""
    g = torch.Generator().manual_seed(int(seed))
    u = torch.randn(shape_u, dtype=F64, generator=g)
    v = torch.randn(shape_v, dtype=F64, generator=g)
    return (0.5 + 0.1 * u).to(device), (0.1 * v).to(device)


def _rhs(case, seed, device):
    """Right-hand side of a Poisson solve: the divergence that a predictor leaves, smooth and rough parts."""
    nx, ny = case["nx"], case["ny"]
    g = torch.Generator().manual_seed(int(seed))
    b = torch.randn((nx, ny), dtype=F64, generator=g)
    u, v = _velocity(nx, ny, *_extent(case), seed)
    smooth = (u[1:] * u[:-1]) + (v[:, 1:] * v[:, :-1])
    return (smooth / smooth.abs().max() + 0.05 * b).to(device)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.kind = case, case["kind"]
    if s.kind == "batch":
        from pycfd_b200.batch import BatchedSolver, BatchOptions, ConcurrentBatch
        n, re, lid = _batch_problems(case, seed)
        cfgs = [SimulationConfig(nx=m, ny=m, re=float(r), u_ref=float(w), dt=1.0, t_end=1e9, cfl_max=0.5,
                                 pressure_solver="mgcg", poisson_tol=TOL, boundary_config=_walls("cavity", float(w)))
                for m, r, w in zip(n, re, lid)]
        opts = BatchOptions(precision=case["precision"])
        if case["tuned"]:
            opts = BatchOptions(precision=case["precision"], inner_tol=1e-3, fused_restriction=True)
        if case["parts"] > 1:
            s.engine = ConcurrentBatch(cfgs, opts, parts=case["parts"])   # starts from rest
            s.pools = [p for part in s.engine.parts for p in part._pools]
        else:
            init = [_velocity(m, m, 1.0, 1.0, seed, k, device="cuda") for k, m in enumerate(n)]
            s.engine = BatchedSolver(cfgs, opts, u_init=[u for u, _ in init], v_init=[v for _, v in init])
            s.pools = list(s.engine._pools)
        return s
    if s.kind == "adjoint":
        from pycfd_b200.adjoint import AdjointCavity, Geometry, MultigridSolve
        cav = _cavity(case, AdjointCavity)
        s.geometry = Geometry(cav, device="cuda")
        s.solve = MultigridSolve(cav.n, tol=cav.tol)
        s.theta, s.radius = (t.cuda() for t in _controls(seed))
        return s
    from pycfd_b200.mesh import StructuredMesh
    from pycfd_b200.obstacles import circle_mask
    from pycfd_b200.simulation import Simulation
    from pycfd_b200.solver import GpuOptions, ProjectionSolver
    if s.kind == "solve":
        s.solver = ProjectionSolver(_config(case))
        s.rhs = _rhs(case, seed, "cuda")
        return s
    if s.kind == "stencil":
        s.solver = ProjectionSolver(_config(dict(case, solver="cg")))
        m = s.solver.mesh
        s.u, s.v = _fields(seed, m.u_shape, m.v_shape, "cuda")
        return s
    cfg = _config(case)
    u, v = _single_init(case, seed, "cuda")
    if s.kind == "run":
        s.sim = Simulation(cfg, u_init=u, v_init=v)
        s.fields = s.sim.fields
        return s
    body = None
    mesh = StructuredMesh.from_config(cfg)
    if case["flow"] in ("cylinder", "stretched"):
        body = circle_mask(mesh, (cfg.lx / 4, cfg.ly / 2), 0.05 if case["flow"] == "cylinder" else 0.1)
    solver = ProjectionSolver(cfg, mesh, body, options=GpuOptions(precision=case["precision"]))
    s.solver, s.dt = solver, cfg.dt
    s.fields = solver.initialize(u, v)
    return s


def _cavity(case, cls):
    return cls(n=case["n"], steps=case["steps"], dt=0.15 / case["n"], re=400.0, modes=32, checkpoint=2)


def _controls(seed):
    rng = np.random.default_rng([int(seed), 5])
    theta = 0.05 * rng.standard_normal(32) / np.arange(1, 33)
    return torch.tensor(theta, dtype=F64), torch.tensor(0.08 + 0.01 * rng.uniform(-1, 1), dtype=F64)


def run(s):
    if s.kind == "batch":
        s.engine.step(1)
        return s.pools
    if s.kind == "adjoint":
        from pycfd_b200.adjoint import objective_fn
        theta, radius = s.theta.clone().requires_grad_(True), s.radius.clone().requires_grad_(True)
        J = objective_fn(theta, radius, s.geometry, s.solve)
        J.backward()
        return {"J": J.detach(), "theta": theta.grad, "radius": radius.grad}
    if s.kind == "solve":
        return s.solver.pressure_solver.solve(s.rhs)
    if s.kind == "stencil":
        ru, rv = s.solver.momentum_rhs(s.u, s.v, s.case["blend"])
        return ru, rv, s.solver.divergence(s.u, s.v)
    if s.kind == "run":
        r = s.sim.stepper.run(s.fields, max_steps=s.case["steps"])
        return {"u": r.fields.u, "v": r.fields.v, "p": r.fields.p, "t": r.fields.t,
                "energy": np.array(r.history["kinetic_energy"])}
    f = s.solver.step(s.fields, s.dt) if s.kind == "step" else s.solver.advance(s.fields, s.dt)
    return f.u, f.v, f.p


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: a step reads the velocity and writes the velocity and the pressure; each
    projection of it reads and writes the solver's vectors once per iteration (the
    method the caller selects): 11 MG-PCG iterations over all levels (the two CG
    kernels and one V-cycle: 9 values per row), or about 4.4 Jacobi-CG iterations per
    cell of the longer side (8 values per cell)."""
    k = case["kind"]
    if k == "stencil":
        return {"bytes": 8 * 5 * case["nx"] * case["ny"], "flops": 90 * case["nx"] * case["ny"]}
    if k == "batch":
        cells = sum(m * m for m in _batch_problems(case, 0)[0])
    elif k == "adjoint":
        cells = case["n"] ** 2
    else:
        cells = case["nx"] * case["ny"]
    s = 4 if case.get("precision") == "mixed" else 8
    if case.get("solver") == "cg":
        its = 4.4 * max(case["nx"], case["ny"])
        solve, flops = its * 8 * 8 * cells, its * 24 * cells
    else:
        solve, flops = MG_ITERATIONS * LEVEL_SUM * 9 * s * cells, MG_ITERATIONS * 130 * cells
    if k == "solve":
        return {"bytes": solve + 16 * cells, "flops": flops}
    if k == "adjoint":   # 3 solves per step forward twice and backward once, and the two initial projections
        solves = 3 * case["steps"] * 4 + 4
        return {"bytes": solves * (solve + 40 * cells), "flops": solves * (flops + 120 * cells)}
    steps = case["steps"] if k == "run" else 1
    return {"bytes": steps * (3 * solve + 40 * cells), "flops": steps * (3 * flops + 3 * 120 * cells)}


# ---------------------------------------------------------------------------
# the same in plain float64 arithmetic (uniform grids, no obstacle)
# ---------------------------------------------------------------------------
def _momentum(u, v, dx, dy, nu, blend=0.0):
    """Advection (central, with a donor-cell part) and diffusion on all u and v faces;
    arrays (..., nx+3, ny+2) and (..., nx+2, ny+3)."""
    c, e, w = u[..., 1:-1, 1:-1], u[..., 2:, 1:-1], u[..., :-2, 1:-1]
    n, s = u[..., 1:-1, 2:], u[..., 1:-1, :-2]
    vt, vb = 0.5 * (v[..., :-1, 2:-1] + v[..., 1:, 2:-1]), 0.5 * (v[..., :-1, 1:-2] + v[..., 1:, 1:-2])
    ur, ul, ut, ub = 0.5 * (c + e), 0.5 * (w + c), 0.5 * (c + n), 0.5 * (s + c)
    a = (ur * ur - ul * ul) / dx + (ut * vt - ub * vb) / dy
    if blend:
        a = a + blend / dx * 0.5 * (ur.abs() * (c - e) - ul.abs() * (w - c))
        a = a + blend / dy * 0.5 * (vt.abs() * (c - n) - vb.abs() * (s - c))
    ru = -a + nu * ((w - 2 * c + e) / dx ** 2 + (s - 2 * c + n) / dy ** 2)
    c, n, s = v[..., 1:-1, 1:-1], v[..., 1:-1, 2:], v[..., 1:-1, :-2]
    e, w = v[..., 2:, 1:-1], v[..., :-2, 1:-1]
    ur, ul = 0.5 * (u[..., 2:-1, :-1] + u[..., 2:-1, 1:]), 0.5 * (u[..., 1:-2, :-1] + u[..., 1:-2, 1:])
    vr, vl, vt, vb = 0.5 * (c + e), 0.5 * (w + c), 0.5 * (c + n), 0.5 * (s + c)
    a = (ur * vr - ul * vl) / dx + (vt * vt - vb * vb) / dy
    if blend:
        a = a + blend / dy * 0.5 * (vt.abs() * (c - n) - vb.abs() * (s - c))
        a = a + blend / dx * 0.5 * (ur.abs() * (c - e) - ul.abs() * (w - c))
    return ru, -a + nu * ((w - 2 * c + e) / dx ** 2 + (s - 2 * c + n) / dy ** 2)


def _div(u, v, dx, dy):
    return ((u[..., 2:-1, 1:-1] - u[..., 1:-2, 1:-1]) / dx + (v[..., 1:-1, 2:-1] - v[..., 1:-1, 1:-2]) / dy)


def _poisson(b, dx, dy, periodic):
    """Mean-free solution of the five-point system by FFT (a closed box by even extension)."""
    nx, ny = b.shape[-2:]
    if not periodic:
        b = torch.cat([b, b.flip(-2)], -2)
        b = torch.cat([b, b.flip(-1)], -1)
    mx, my = b.shape[-2:]
    kx = torch.arange(mx, dtype=F64, device=b.device)
    ky = torch.arange(my // 2 + 1, dtype=F64, device=b.device)
    lam = (-4 * torch.sin(math.pi * kx / mx) ** 2 / dx ** 2)[:, None] \
        + (-4 * torch.sin(math.pi * ky / my) ** 2 / dy ** 2)[None, :]
    lam[0, 0] = 1.0
    f = torch.fft.rfft2(b) / lam
    keep = torch.ones_like(lam)
    keep[0, 0] = 0.0
    return torch.fft.irfft2(f * keep, s=(mx, my))[..., :nx, :ny]


class _Box:
    """A closed box with a moving lid, or a doubly periodic one; leading dimensions of the
    arrays are independent problems, ``lid`` and ``nu`` broadcast against them."""

    def __init__(self, nx, ny, lx, ly, nu, lid=None, chi=None):
        self.nx, self.ny, self.dx, self.dy, self.nu = nx, ny, lx / nx, ly / ny, nu
        self.lid, self.chi = lid, chi      # lid None: periodic
        lo = 1 if lid is None else 2
        self.su = (..., slice(lo, nx + 1), slice(1, ny + 1))
        self.sv = (..., slice(1, nx + 1), slice(lo, ny + 1))

    def walls(self, u, v):
        nx, ny = self.nx, self.ny
        u, v = u.clone(), v.clone()
        if self.lid is None:
            u[..., nx + 1, :] = u[..., 1, :]
            u[..., 0, :] = u[..., nx, :]
            u[..., nx + 2, :] = u[..., 2, :]
            v[..., 0, :] = v[..., nx, :]
            v[..., nx + 1, :] = v[..., 1, :]
            v[..., ny + 1] = v[..., 1]
            v[..., 0] = v[..., ny]
            v[..., ny + 2] = v[..., 2]
            u[..., 0] = u[..., ny]
            u[..., ny + 1] = u[..., 1]
            return u, v
        u[..., 1, :] = 0.0
        u[..., 0, :] = -u[..., 2, :]
        v[..., 0, :] = -v[..., 1, :]
        u[..., nx + 1, :] = 0.0
        u[..., nx + 2, :] = -u[..., nx, :]
        v[..., nx + 1, :] = -v[..., nx, :]
        v[..., 1] = 0.0
        v[..., 0] = -v[..., 2]
        u[..., 0] = -u[..., 1]
        v[..., ny + 1] = 0.0
        v[..., ny + 2] = -v[..., ny]
        u[..., ny + 1] = 2.0 * self.lid - u[..., ny]
        return u, v

    def mask(self, u, v):
        if self.chi is None:
            return u, v
        a, b = u.clone(), v.clone()
        a[self.su] = (1.0 - self.chi[0][self.su]) * u[self.su]
        b[self.sv] = (1.0 - self.chi[1][self.sv]) * v[self.sv]
        return a, b

    def project(self, u, v, dt):
        q = _poisson(_div(u, v, self.dx, self.dy) / dt, self.dx, self.dy, self.lid is None)
        nx, ny = self.nx, self.ny
        if self.lid is None:
            p = torch.cat([q[..., -1:, :], q, q[..., :1, :]], -2)
            p = torch.cat([p[..., -1:], p, p[..., :1]], -1)
        else:
            p = torch.cat([q[..., :1, :], q, q[..., -1:, :]], -2)
            p = torch.cat([p[..., :1], p, p[..., -1:]], -1)
        u, v = u.clone(), v.clone()
        gu = (p[..., 1:, :] - p[..., :-1, :]) / self.dx       # face m between cells m-1 and m (ghosted)
        gv = (p[..., 1:] - p[..., :-1]) / self.dy
        lo = self.su[1].start
        u[self.su] = u[self.su] - dt * gu[..., lo - 1:nx, 1:ny + 1]
        v[self.sv] = v[self.sv] - dt * gv[..., 1:nx + 1, lo - 1:ny]
        return u, v, p

    def close(self, u, v, dt):
        u, v = self.mask(*self.walls(u, v))
        if self.lid is None:
            u, v = self.walls(u, v)
        u, v, p = self.project(u, v, dt)
        return (*self.walls(*self.mask(u, v)), p)

    def initial(self, u0, v0):
        u = torch.zeros(u0.shape[:-2] + (self.nx + 3, self.ny + 2), dtype=F64, device=u0.device)
        v = torch.zeros(v0.shape[:-2] + (self.nx + 2, self.ny + 3), dtype=F64, device=u0.device)
        u[..., 1:self.nx + 2, 1:self.ny + 1] = u0
        v[..., 1:self.nx + 1, 1:self.ny + 2] = v0
        return self.close(u, v, 1.0)

    def substep(self, u, v, dt):
        ru, rv = _momentum(u, v, self.dx, self.dy, self.nu)
        us, vs = u.clone(), v.clone()
        lo = self.su[1].start
        us[self.su] = us[self.su] + dt * ru[..., lo - 1:self.nx, :]
        vs[self.sv] = vs[self.sv] + dt * rv[..., lo - 1:self.ny]
        return self.close(us, vs, dt)

    def step(self, u, v, dt):
        a, b, _ = self.substep(u, v, dt)
        a, b, _ = self.substep(a, b, dt)
        a, b, p = self.substep(0.75 * u + 0.25 * a, 0.75 * v + 0.25 * b, dt)
        return (*self.walls(u / 3.0 + 2.0 / 3.0 * a, v / 3.0 + 2.0 / 3.0 * b), p)

    def adaptive(self, u, v, cfl=0.5):
        um = u[..., 1:self.nx + 2, 1:self.ny + 1].abs().amax((-2, -1), keepdim=True)
        vm = v[..., 1:self.nx + 1, 1:self.ny + 2].abs().amax((-2, -1), keepdim=True)
        visc = 0.8 / (2.0 * self.nu * (1.0 / self.dx ** 2 + 1.0 / self.dy ** 2))
        return torch.minimum(cfl / (um / self.dx + vm / self.dy), visc * torch.ones_like(um)).clamp(max=1.0)


def _parts(cells, parts):
    """Problems per concurrent part, largest first to the part with the fewest cells."""
    out, load = [[] for _ in range(parts)], [0] * parts
    for k in sorted(range(len(cells)), key=lambda k: (-cells[k], k)):
        r = min(range(parts), key=lambda q: (load[q], q))
        out[r].append(k)
        load[r] += cells[k]
    return [sorted(o) for o in out if o]


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    k = case["kind"]
    if k == "batch":
        n, re, lid = _batch_problems(case, seed)
        got = [None] * len(n)
        for m in sorted(set(n)):
            ks = [q for q in range(len(n)) if n[q] == m]
            col = lambda a: torch.tensor([float(a[q]) for q in ks], dtype=F64, device=dev)[:, None, None]  # noqa: E731
            w = col(lid)
            box = _Box(m, m, 1.0, 1.0, w / col(re), lid=w[:, 0])
            init = [_velocity(m, m, 1.0, 1.0, seed, q, device=dev) for q in ks]
            u0, v0 = (torch.stack([t[a] for t in init]) for a in (0, 1))
            rest = 0.0 if case["parts"] > 1 else 1.0   # concurrent parts start from rest
            u, v, _ = box.initial(rest * u0, rest * v0)
            out = box.step(u, v, box.adaptive(u, v))
            for j, q in enumerate(ks):
                got[q] = [t[j].reshape(-1) for t in out]
        return [torch.cat([got[q][a] for q in ks]) for ks in _parts([m * m for m in n], case["parts"])
                for a in range(3)]
    if k == "adjoint":
        from types import SimpleNamespace
        c = _cavity(case, SimpleNamespace)
        n, h = c.n, 1.0 / c.n
        theta, radius = (t.to(dev).requires_grad_(True) for t in _controls(seed))
        xm = (torch.arange(n + 3, dtype=F64, device=dev) - 1.0) * h
        yj = (torch.arange(n + 2, dtype=F64, device=dev) - 0.5) * h
        basis = torch.sin(math.pi * torch.arange(1, 33, dtype=F64, device=dev)[:, None] * xm[None, :])
        chi = [0.5 * (1.0 - torch.tanh((torch.sqrt((a - 0.5)[:, None] ** 2 + (b - 0.3)[None, :] ** 2) - radius)
                                       / (2.0 * h))) for a, b in ((xm, yj), (yj, xm))]
        box = _Box(n, n, 1.0, 1.0, 1.0 / c.re, lid=1.0 + theta @ basis, chi=chi)
        u, v, _ = box.initial(torch.zeros(n + 1, n, dtype=F64, device=dev), torch.zeros(n, n + 1, dtype=F64, device=dev))
        for _ in range(c.steps):
            u, v, _ = box.step(u, v, c.dt)
        uc, vc = 0.5 * (u[1:-2, 1:-1] + u[2:-1, 1:-1]), 0.5 * (v[1:-1, 1:-2] + v[1:-1, 2:-1])
        low = ((torch.arange(n, dtype=F64, device=dev) + 0.5) * h < 0.5).to(F64)
        J = (0.5 * (uc * uc + vc * vc) * low).sum() * h * h
        J.backward()
        return {"J": J.detach(), "theta": theta.grad, "radius": radius.grad}
    nx, ny = case["nx"], case["ny"]
    lx, ly = _extent(case)
    if k == "solve":
        return _poisson(_rhs(case, seed, dev), lx / nx, ly / ny, False)
    if k == "stencil":
        u, v = _fields(seed, (nx + 3, ny + 2), (nx + 2, ny + 3), dev)
        return (*_momentum(u, v, lx / nx, ly / ny, 1.0 / 400.0, case["blend"]), _div(u, v, lx / nx, ly / ny))
    flow = case.get("flow", "cavity")
    if flow not in ("cavity", "periodic"):
        return None
    box = _Box(nx, ny, lx, ly, 1.0 / (100.0 if k == "run" else 400.0), lid=None if flow == "periodic" else 1.0)
    u, v, p = box.initial(*_single_init(case, seed, dev))
    if k != "run":
        return box.step(u, v, _dt(case))
    t, energy = 0.0, []
    for _ in range(case["steps"]):
        dt = box.adaptive(u, v)
        u, v, p = box.step(u, v, dt)
        t += float(dt)
        uc, vc = 0.5 * (u[1:-2, 1:-1] + u[2:-1, 1:-1]), 0.5 * (v[1:-1, 1:-2] + v[1:-1, 2:-1])
        energy.append(float((0.5 * (uc * uc + vc * vc)).sum()) * box.dx * box.dy)
    return {"u": u, "v": v, "p": p, "t": t, "energy": np.array(energy)}
