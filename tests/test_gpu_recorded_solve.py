"""Pressure solves called one by one, past the count after which a solver records its
solve as a graph (needs a B200).

The host loop of the first calls and the recorded loop of the later ones run the same
passes to the same stopping test, so every call on one right-hand side gives the same
bits and the same count, for each warm start and on streams other than the default.
"""

import numpy as np
import pytest

import cases
from pycfd_b200.config import BCKind, BCSpec, SimulationConfig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CALLS = 10   # the first six loop on the host


@pytest.mark.parametrize("nx,ny,kind,precision,bc", [
    (64, 48, "mgcg", "fp64", cases.bcs()), (129, 65, "mgcg", "fp64", cases.PER), (8, 8, "mgcg", "fp64", cases.bcs()),
    (96, 64, "mgcg", "mixed", cases.bcs()), (65, 130, "mgcg", "mixed", cases.PER),
    (64, 64, "multigrid", "fp64", cases.bcs()), (520, 257, "cg", "fp64", cases.bcs(right=("pressure_outlet",)))])
def test_every_call_gives_the_same_bits(nx, ny, kind, precision, bc):
    from pycfd_b200.solver import GpuOptions, ProjectionSolver
    lx, ly = nx / max(nx, ny), ny / max(nx, ny)
    cfg = cases.to_config(dict(nx=nx, ny=ny, lx=lx, ly=ly, re=100.0, pressure_solver=kind, poisson_tol=1e-8,
                               boundary_config=bc), SimulationConfig, BCSpec, BCKind)
    s = ProjectionSolver(cfg, options=GpuOptions(precision=precision))
    rng = np.random.default_rng(nx + ny)
    rhs, other = rng.standard_normal((2, nx, ny))
    start = 0.1 * rng.standard_normal((nx, ny))
    p = s.pressure_solver
    seen = {}
    streams = [torch.cuda.current_stream(), torch.cuda.Stream()]
    for call in range(CALLS):
        for name, b, p0 in (("cold", rhs, None), ("warm", rhs, start), ("other", other, None)):
            with torch.cuda.stream(streams[call % 2]):
                x = p.solve(b, p0).cpu().numpy()
            streams[call % 2].synchronize()
            got = (p.last_iterations, x)
            want = seen.setdefault(name, got)
            assert got[0] == want[0] and np.array_equal(got[1], want[1]), (name, call)
