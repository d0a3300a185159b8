"""Bent one-cell channels (needs a B200): masks whose coarse levels take the row widths of
the usual level-0 product, on row patterns against the stored level operators."""

import numpy as np
import pytest

import cases
from oracle.poisson import assemble_poisson
from pycfd_b200.config import BCKind, BCSpec, SimulationConfig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 1e-10


def channel(nx, ny, w, i, j):
    solid = np.ones((nx, ny), bool)
    solid[i:i + w, j:] = False
    solid[i:, j:j + w] = False
    return solid


def _cfg(nx, ny, **kw):
    return cases.to_config(dict(nx=nx, ny=ny, lx=nx / 64.0, ly=ny / 64.0, re=100.0, pressure_solver="mgcg",
                                poisson_tol=TOL, boundary_config=cases.bcs(), **kw),
                           SimulationConfig, BCSpec, BCKind)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,w,i,j", [(135, 145, 1, 3, 6), (151, 177, 1, 111, 110)])
def test_solver_of_a_bent_channel(nx, ny, w, i, j, precision):
    from pycfd_b200 import _lib
    from pycfd_b200.solver import GpuOptions, ProjectionSolver
    cfg, solid, L = _cfg(nx, ny), channel(nx, ny, w, i, j), _lib.load()
    rng = np.random.default_rng(nx)
    r, rhs = rng.standard_normal((2, nx, ny))
    r[solid] = 0.0
    sysm = assemble_poisson(nx, ny, cfg.lx / nx, cfg.ly / ny, False, False, solid, None)
    b = rhs.ravel().copy()
    b[~sysm.fluid] = 0.0
    if sysm.singular:
        b[sysm.fluid] -= b[sysm.fluid].mean()
    z, its = [], []
    for products in (True, False):   # row patterns; the stored operators level by level
        s = ProjectionSolver(cfg, obstacle=solid, options=GpuOptions(
            precision=precision, fused_restriction=products, coarse_tail=products))
        rd = torch.as_tensor(r, device="cuda")
        out = torch.empty_like(rd)
        _lib.check(L.pycfd_mg_apply(s._h, _lib.ptr(rd), _lib.ptr(out), None))
        z.append(out.cpu().numpy())
        p = s.pressure_solver.solve(rhs).cpu().numpy()
        assert s.last_stats.status == 0
        assert np.linalg.norm(b - sysm.A @ p.ravel()) < 10 * TOL * np.linalg.norm(b)
        its.append(s.pressure_solver.last_iterations)
    # a few hundred products per row and level, each rounded once
    assert np.abs(z[0] - z[1]).max() < 1e-12 * np.abs(z[1]).max()
    assert abs(its[0] - its[1]) <= 2, its


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_of_bent_channels(precision):
    """The projection of a random velocity, three problems of each channel (a group of
    several problems and its remainder) and one open cavity, against one problem per
    block, which keeps the stored operators.  (No steps: the flow of a closed channel one
    cell wide is zero, and what is left after the projection is rounding.)"""
    from pycfd_b200.batch import BatchedSolver, BatchOptions
    shapes = [(51, 71, 1, 14, 23)] * 3 + [(13, 78, 1, 10, 0)] * 3 + [(32, 32, 0, 0, 0)]
    cfgs, bodies, u0 = [], [], []
    rng = np.random.default_rng(3)
    for nx, ny, w, i, j in shapes:
        cfgs.append(_cfg(nx, ny, adaptive_dt=False, dt=1e-4, t_end=10.0))
        bodies.append(channel(nx, ny, w, i, j) if w else None)
        u0.append(rng.standard_normal((nx + 1, ny)))
    out = []
    for group in (8, 1):
        b = BatchedSolver(cfgs, BatchOptions(precision=precision, ell_group=group), obstacles=bodies, u_init=u0)
        st = b.status()
        assert not st["status"].any()
        out.append([f.numpy() for f in b.fields] + [st["iterations"]])
    assert np.abs(out[0][-1] - out[1][-1]).max() <= 2, (out[0][-1], out[1][-1])
    for x, y, u in zip(out[0][:-1], out[1][:-1], u0):
        # both project u to 1e-10; the pressure inherits the solve's tolerance
        scale = (np.abs(u).max(), np.abs(u).max(), np.abs(y[2]).max())
        for p, q, size in zip(x, y, scale):
            assert np.abs(p - q).max() <= 1e-8 * size
