"""Batches whose structures take different forms of the V-cycle (needs a B200): a problem's
results must not depend on the problems beside it, bit for bit."""

import numpy as np
import pytest

import cases
from pycfd_b200.config import BCKind, BCSpec, SimulationConfig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LID = cases.bcs(top=("moving_wall", 1.0))


def pegs(n, seed=0):
    """One solid cell at a random place of every 4 x 4 block (rows of fluid between them):
    nearly every row of a coarse level has a pattern of its own."""
    rng = np.random.default_rng(seed)
    solid = np.zeros((n, n), bool)
    for a in range(0, n - 3, 4):
        for b in range(0, n - 3, 4):
            solid[a + rng.integers(3), b + rng.integers(3)] = True
    return solid


def _cfg(n, re):
    return cases.to_config(dict(nx=n, ny=n, re=re, pressure_solver="mgcg", poisson_tol=1e-10, adaptive_dt=False,
                                dt=1e-4, t_end=10.0, boundary_config=LID), SimulationConfig, BCSpec, BCKind)


def _run(cfgs, bodies, options, steps=2):
    from pycfd_b200.batch import BatchedSolver
    b = BatchedSolver(cfgs, options, obstacles=bodies)
    b.step(steps)
    st = b.status()
    assert not st["status"].any() and not st["frozen"].any()
    return [(*f.numpy(), it) for f, it in zip(b.fields, st["iterations"])]


@pytest.mark.parametrize("precision,fused", [("fp64", False), ("mixed", False), ("mixed", True)])
def test_a_structure_without_patterns_leaves_the_others_alone(precision, fused):
    """A mask with more patterns than a table can name (560 x 560 pegs) beside cavities
    with and without a dense tail."""
    from pycfd_b200.batch import BatchOptions
    opts = BatchOptions(precision=precision, fused_restriction=fused)
    cfgs = [_cfg(560, 100.0), _cfg(50, 150.0), _cfg(50, 200.0), _cfg(16, 100.0)]
    bodies = [pegs(560), None, None, None]
    together = _run(cfgs, bodies, opts)
    apart = _run(cfgs[:1], bodies[:1], opts) + _run(cfgs[1:], bodies[1:], opts)
    for k, (a, b) in enumerate(zip(together, apart)):
        assert a[3] == b[3], k
        for p, q in zip(a[:3], b[:3]):
            assert np.array_equal(p, q), k


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_more_structures_than_the_hierarchy_cache_keeps(precision):
    """Twelve masks of their own in one batch, against each mask alone."""
    from pycfd_b200.batch import BatchOptions
    opts = BatchOptions(precision=precision)
    cfgs = [_cfg(64, 100.0 + 5 * k) for k in range(12)]
    bodies = [pegs(64, seed=k) for k in range(12)]
    for k, (a, b) in enumerate(zip(_run(cfgs, bodies, opts),
                                   (_run(cfgs[k:k + 1], bodies[k:k + 1], opts)[0] for k in range(12)))):
        assert a[3] == b[3], k
        for p, q in zip(a[:3], b[:3]):
            assert np.array_equal(p, q), k
