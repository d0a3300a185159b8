"""Row patterns on grids a few cells wide along either axis (needs a B200): the products'
tiles narrow with the grid; one cycle against the stored level operators."""

import numpy as np
import pytest

import cases
from pycfd_b200.config import BCKind, BCSpec, SimulationConfig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 33), (60000, 64), (3, 40000), (2400, 8), (2, 80000)])
def test_divergence_covers_every_cell(nx, ny):
    """Fewer and more cells than the launch has threads, along either axis."""
    from pycfd_b200 import _lib
    L = _lib.load()
    u = torch.randn(nx + 3, ny + 2, dtype=torch.float64, device="cuda")
    v = torch.randn(nx + 2, ny + 3, dtype=torch.float64, device="cuda")
    out = torch.full((nx, ny), float("nan"), dtype=torch.float64, device="cuda")
    _lib.check(L.pycfd_divergence(_lib.ptr(u), _lib.ptr(v), nx, ny, 0.25, 0.5, _lib.ptr(out), None))
    want = (u[2:nx + 2, 1:ny + 1] - u[1:nx + 1, 1:ny + 1]) / 0.25 + (v[1:nx + 1, 2:ny + 2] - v[1:nx + 1, 1:ny + 1]) / 0.5
    torch.cuda.synchronize()
    assert torch.equal(out, want)   # powers of two divide exactly; one sum


@pytest.mark.parametrize("nx,ny", [(300, 4), (1000, 5), (401, 8), (257, 16), (2000, 17), (5, 700), (4, 2001), (40001, 4)])
def test_cycle_on_a_thin_grid(nx, ny):
    from pycfd_b200 import _lib
    from pycfd_b200.solver import GpuOptions, ProjectionSolver
    cfg = cases.to_config(dict(nx=nx, ny=ny, lx=nx / 64.0, ly=ny / 64.0, re=100.0, pressure_solver="mgcg",
                               poisson_tol=1e-10, boundary_config=cases.bcs(right=("pressure_outlet",))),
                          SimulationConfig, BCSpec, BCKind)
    r = np.random.default_rng(nx + ny).standard_normal((nx, ny))
    z = []
    for products in (True, False):
        s = ProjectionSolver(cfg, options=GpuOptions(fused_restriction=products, coarse_tail=products))
        assert (s.form()["pattern_levels"] > 0) == products
        rd = torch.as_tensor(r, device="cuda")
        out = torch.empty_like(rd)
        _lib.check(_lib.load().pycfd_mg_apply(s._h, _lib.ptr(rd), _lib.ptr(out), None))
        z.append(out.cpu().numpy())
    # a few hundred products per row and level, each rounded once
    assert np.abs(z[0] - z[1]).max() < 1e-12 * np.abs(z[1]).max()
