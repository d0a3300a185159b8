"""The V-cycle as products of row patterns against the general level operators (needs a B200).

Both are the same linear map, so one cycle agrees to rounding and solves agree to
the tolerance; the shapes cover the sizes where the tables can go wrong: odd extents on
either axis, both seams, Dirichlet edges, bodies, semi-coarsened anisotropic cells, a
level of one row, and levels whose rows end inside a block.
"""

import numpy as np
import pytest

import cases
from oracle.projection import circle_mask_oracle
from pycfd_b200.config import BCKind, BCSpec, SimulationConfig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WALLS = cases.bcs(top=("moving_wall", 1.0))
SEAM_X = cases.bcs(left=("periodic",), right=("periodic",))
OUT = cases.bcs(right=("pressure_outlet", 0.0, "uniform", 0.2))


def _cfg(nx, ny, bc, ly=None, **kw):
    d = dict(nx=nx, ny=ny, lx=1.0, ly=ny / nx if ly is None else ly, re=100.0, pressure_solver="mgcg",
             poisson_tol=1e-11, boundary_config=bc, **kw)
    return cases.to_config(d, SimulationConfig, BCSpec, BCKind)


@pytest.mark.parametrize("nx,ny,bc,ly,body", [
    (64, 64, WALLS, None, False), (101, 77, WALLS, None, False), (96, 130, cases.PER, None, True),
    (67, 90, SEAM_X, None, True), (150, 61, OUT, None, True), (128, 64, WALLS, 0.1, False),
    (300, 5, WALLS, None, False), (257, 255, cases.PER, None, False)])
def test_pattern_cycle_is_the_level_by_level_cycle(nx, ny, bc, ly, body):
    from pycfd_b200 import _lib
    from pycfd_b200.solver import GpuOptions, ProjectionSolver
    cfg = _cfg(nx, ny, bc, ly)
    solid = circle_mask_oracle(nx, ny, cfg.lx, cfg.ly, (0.4 * cfg.lx, 0.5 * cfg.ly), 0.2 * min(cfg.lx, cfg.ly)) \
        if body else None
    L = _lib.load()
    r = np.random.default_rng(nx + ny).standard_normal((nx, ny))
    if solid is not None:
        r[solid] = 0.0
    z = []
    for fused in (True, False):   # the products; the stored operators level by level
        s = ProjectionSolver(cfg, obstacle=solid, options=GpuOptions(fused_restriction=fused, coarse_tail=fused))
        rd = torch.as_tensor(r, device="cuda")
        out = torch.empty_like(rd)
        _lib.check(L.pycfd_mg_apply(s._h, _lib.ptr(rd), _lib.ptr(out), None))
        z.append(out.cpu().numpy())
    # a few hundred products per row and level, each rounded once
    assert np.abs(z[0] - z[1]).max() < 1e-12 * np.abs(z[1]).max()


@pytest.mark.parametrize("precision,bound", [("fp64", 1e-9), ("mixed", 1e-9)])
def test_batch_on_patterns_matches_the_general_operators(precision, bound):
    """Odd and even cavities, a seam, a Dirichlet outlet with a body and an untailed small
    grid in one batch, 1 to 9 problems per structure, against one problem per block
    (ell_group 1), which keeps the stored operators."""
    from pycfd_b200.batch import BatchedSolver, BatchOptions
    shapes = [(16, 16, WALLS)] * 2 + [(50, 50, WALLS)] * 9 + [(77, 101, WALLS)] * 3 + [(64, 96, SEAM_X), (90, 60, OUT)]
    cfgs, bodies = [], []
    for k, (nx, ny, bc) in enumerate(shapes):
        cfgs.append(_cfg(nx, ny, bc, adaptive_dt=False, dt=1e-3, t_end=10.0).replace(re=100.0 + 20 * k))
        body = bc is OUT
        bodies.append(circle_mask_oracle(nx, ny, cfgs[-1].lx, cfgs[-1].ly, (0.5, 0.3), 0.1) if body else None)
    out = []
    for group in (8, 1):
        b = BatchedSolver(cfgs, BatchOptions(precision=precision, ell_group=group), obstacles=bodies)
        b.step(3)
        assert not b.status()["status"].any()
        out.append([f.numpy() for f in b.fields])
    for x, y in zip(*out):
        # the outlet problem has no inflow: its velocities are what the solve of its
        # pressure (p_ref 0.2) leaves, so a problem's fields are measured by its largest
        scale = max(np.abs(q).max() for q in y)
        for p, q in zip(x, y):
            assert np.abs(p - q).max() <= bound * scale
