"""Batches of thousands of equal small problems (needs a B200): every problem of a
structure must be solved, however many share it."""

import numpy as np
import pytest

import cases
from pycfd_b200.config import BCKind, BCSpec, SimulationConfig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _cfg(n):
    return cases.to_config(dict(nx=n, ny=n, re=100.0, pressure_solver="mgcg", poisson_tol=1e-10, adaptive_dt=False,
                                dt=2e-3, t_end=10.0, boundary_config=cases.bcs(top=("moving_wall", 1.0))),
                           SimulationConfig, BCSpec, BCKind)


def _equal_problems(n, count, options):
    from pycfd_b200.batch import BatchedSolver
    b = BatchedSolver([_cfg(n)] * count, options)
    b.step(2)
    st = b.status()
    assert not st["status"].any() and not st["frozen"].any()
    assert (st["iterations"] == st["iterations"][0]).all() and (st["t"] == st["t"][0]).all()
    for pool, shape in zip(b._pools, (f.shape for f in (b.fields[0].u, b.fields[0].v, b.fields[0].p))):
        every = pool.view(count, *shape)
        assert torch.isfinite(every).all() and every[0].abs().max() > 0
        assert (every == every[0]).all()   # equal problems, equal bits
    return b


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_more_problems_than_64_column_tiles(precision):
    """2100 problems closed by one dense tail: 66 column tiles of 32 problems."""
    from pycfd_b200.batch import BatchOptions
    _equal_problems(20, 2100, BatchOptions(precision=precision, tail_ratio=None))


@pytest.mark.parametrize("n,precision", [(20, "fp64"), (10, "fp64"), (10, "mixed")])
def test_more_problems_than_1024_groups_of_four(n, precision):
    """4100 problems of one structure: a tail on the 20 x 20 grid, none on the 10 x 10 one."""
    from pycfd_b200.batch import BatchOptions
    _equal_problems(n, 4100, BatchOptions(precision=precision, tail_ratio=None if n == 20 else 16.0))
