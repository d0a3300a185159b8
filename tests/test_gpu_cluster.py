"""Jacobi-CG solves of small grids as one cluster launch (needs a B200).

Every band layout the rule can pick -- one row per CTA, fewer rows than CTAs, bands
of unequal height, each count of cells per thread, the largest grid that fits and the
first that does not -- against the assembled matrix and against the one-kernel-per-
phase passes of the persistent form on the same right-hand side.
"""

import numpy as np
import pytest

import cases
from oracle.poisson import assemble_poisson
from oracle.projection import circle_mask_oracle
from pycfd_b200.config import BCKind, BCSpec, SimulationConfig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WALLS = cases.bcs()
MIXED = cases.bcs(bottom=("periodic",), top=("periodic",), right=("pressure_outlet", 0.0, "uniform", 0.3))
SIDE = cases.bcs(left=("periodic",), right=("periodic",), top=("pressure_outlet",))
TOL = 1e-10


@pytest.mark.parametrize("nx,ny,bc,body", [
    (4, 4, WALLS, False), (5, 33, cases.PER, False), (16, 16, WALLS, False), (17, 40, cases.PER, False),
    (24, 8, SIDE, False), (64, 64, WALLS, True), (97, 61, MIXED, True), (200, 150, WALLS, False),
    (6, 1300, MIXED, False), (300, 96, cases.PER, True), (256, 250, WALLS, False), (500, 190, SIDE, False),
    (512, 256, WALLS, False), (512, 257, WALLS, False), (15, 8192, WALLS, False)])
def test_cluster_cg_solves_the_assembled_system(nx, ny, bc, body):
    from pycfd_b200.solver import GpuOptions, ProjectionSolver
    lx, ly = nx / max(nx, ny), ny / max(nx, ny)
    cfg = cases.to_config(dict(nx=nx, ny=ny, lx=lx, ly=ly, re=100.0, pressure_solver="cg", poisson_tol=TOL,
                               boundary_config=bc), SimulationConfig, BCSpec, BCKind)
    solid = circle_mask_oracle(nx, ny, lx, ly, (0.4 * lx, 0.5 * ly), 0.15 * min(lx, ly)) if body else None
    s = ProjectionSolver(cfg, obstacle=solid)
    rng = np.random.default_rng(nx * 1000 + ny)
    rhs = rng.standard_normal((nx, ny))
    dirichlet = {w: sp[3] if len(sp) > 3 else 0.0 for w, sp in bc.items() if sp[0] == "pressure_outlet"}
    per_x, per_y = bc["left"][0] == "periodic", bc["bottom"][0] == "periodic"
    sysm = assemble_poisson(nx, ny, lx / nx, ly / ny, per_x, per_y, solid, dirichlet or None)
    b = rhs.ravel() + sysm.bc_rhs
    b[~sysm.fluid] = 0.0
    if sysm.singular:
        b[sysm.fluid] -= b[sysm.fluid].mean()
    general = ProjectionSolver(cfg, obstacle=solid, options=GpuOptions(persistent_solve=True))
    want = general.pressure_solver.solve(rhs).cpu().numpy()
    its = general.pressure_solver.last_iterations
    for p0 in (None, 0.9 * want):
        p = s.pressure_solver.solve(rhs, p0).cpu().numpy()
        assert s.last_stats.status == 0
        # the recurrence residual is below tol; the true one may drift by its rounding, kappa eps
        assert np.linalg.norm(b - sysm.A @ p.ravel()) < 10 * TOL * np.linalg.norm(b)
        if p0 is None:   # the same recurrence: only the dot products' order differs
            assert abs(s.pressure_solver.last_iterations - its) <= max(3, 0.03 * its)
            again = s.pressure_solver.solve(rhs).cpu().numpy()
            assert np.array_equal(p, again)
