"""Structures without a dense tail under the pattern products (needs a B200): closed per
problem on their coarsest level, alone and beside tailed ones, against one problem per
block, which keeps the stored operators and closes in the same way."""

import numpy as np
import pytest

import cases
from pycfd_b200.config import BCKind, BCSpec, SimulationConfig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LID = cases.bcs(top=("moving_wall", 1.0))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shapes,tail", [([(10, 10)] * 3, True), ([(16, 16), (13, 24), (32, 32), (24, 24)] * 2, True),
                                         ([(10, 10), (50, 50), (24, 24), (64, 64)], True),
                                         ([(50, 50), (64, 64)], False)])
def test_untailed_structures(shapes, tail, precision):
    from pycfd_b200.batch import BatchedSolver, BatchOptions
    cfgs = [cases.to_config(dict(nx=nx, ny=ny, lx=nx / 32.0, ly=ny / 32.0, re=100.0 + 10 * k, pressure_solver="mgcg",
                                 poisson_tol=1e-10, adaptive_dt=False, dt=1e-3, t_end=10.0, boundary_config=LID),
                            SimulationConfig, BCSpec, BCKind) for k, (nx, ny) in enumerate(shapes)]
    out = []
    for group in (8, 1):
        b = BatchedSolver(cfgs, BatchOptions(precision=precision, ell_group=group, coarse_tail=tail))
        b.step(3)
        st = b.status()
        assert not st["status"].any() and not st["frozen"].any()
        out.append([f.numpy() for f in b.fields] + [st["iterations"]])
    # the same cycle to rounding: a pass more or less per solve (three per step) at most
    assert np.abs(out[0][-1] - out[1][-1]).max() <= 3, (out[0][-1], out[1][-1])
    for x, y in zip(out[0][:-1], out[1][:-1]):
        for p, q in zip(x, y):
            assert np.abs(p - q).max() <= 1e-8 * max(np.abs(f).max() for f in y)
