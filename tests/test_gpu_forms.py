"""Which form of a solve is in force, and its results there (needs a B200): the other tests
compare results, which hold too where a rule falls back; here the form is asserted first.
"""

import numpy as np
import pytest

import cases
from pycfd_b200.config import BCKind, BCSpec, SimulationConfig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LID = cases.bcs(top=("moving_wall", 1.0))


def _cfg(nx, ny, bc=LID, **kw):
    d = dict(nx=nx, ny=ny, lx=nx / max(nx, ny), ly=ny / max(nx, ny), re=100.0, pressure_solver="mgcg",
             poisson_tol=1e-10, boundary_config=bc)
    return cases.to_config({**d, **kw}, SimulationConfig, BCSpec, BCKind)


def _solver(cfg, **options):
    from pycfd_b200.solver import GpuOptions, ProjectionSolver
    return ProjectionSolver(cfg, options=GpuOptions(**options))


def _cycle(s, r):
    from pycfd_b200 import _lib
    rd = torch.as_tensor(r, device="cuda")
    out = torch.empty_like(rd)
    _lib.check(_lib.load().pycfd_mg_apply(s._h, _lib.ptr(rd), _lib.ptr(out), None))
    return out.cpu().numpy()


@pytest.mark.parametrize("nx,ny,bc,tiles", [(64, 48, LID, 1), (389, 389, LID, 2), (523, 311, cases.PER, 2),
                                            (640, 480, cases.bcs(right=("pressure_outlet",)), 3)])
def test_single_cycle_on_patterns(nx, ny, bc, tiles):
    """One wave of blocks is 592 tiles of 8 x 32 cells: the larger grids walk 2 and 3 each."""
    s = _solver(_cfg(nx, ny, bc))
    form = s.form()
    assert form["pattern_levels"] > 0 and form["up_tiles"] == tiles and form["cluster_ctas"] == 0
    g = _solver(_cfg(nx, ny, bc), fused_restriction=False, coarse_tail=False)
    assert g.form()["pattern_levels"] == 0
    r = np.random.default_rng(nx).standard_normal((nx, ny))
    a, b = _cycle(s, r), _cycle(g, r)
    assert np.abs(a - b).max() < 1e-12 * np.abs(b).max()


def test_forms_that_keep_stored_operators():
    assert _solver(_cfg(96, 96), fused_restriction=False).form()["pattern_levels"] == 0
    assert _solver(_cfg(96, 96, mg_sweeps=2)).form()["pattern_levels"] == 0
    assert _solver(_cfg(96, 96), persistent_solve=True).form()["pattern_levels"] == 0


def test_cluster_and_recorded_solves():
    cg = _solver(_cfg(64, 64, pressure_solver="cg", poisson_tol=1e-8))
    assert cg.form()["cluster_ctas"] > 0
    assert _solver(_cfg(512, 257, pressure_solver="cg")).form()["cluster_ctas"] == 0
    mg = _solver(_cfg(64, 64))
    rhs = np.random.default_rng(0).standard_normal((64, 64))
    seen = []
    for _ in range(8):
        mg.pressure_solver.solve(rhs)
        cg.pressure_solver.solve(rhs)
        seen.append(mg.form()["recorded_solves"])
    assert seen == [0] * 6 + [1] * 2 and cg.form()["recorded_solves"] == 0
    mg.pressure_solver.solve(rhs, 0.1 * rhs)   # a warm start records its own
    assert mg.form()["recorded_solves"] == 2


@pytest.mark.parametrize("precision,count,group,up", [("mixed", 243, 8, 4), ("mixed", 122, 4, 2), ("mixed", 63, 2, 1),
                                                      ("mixed", 9, 1, 1), ("fp64", 243, 4, 2), ("fp64", 70, 2, 1)])
def test_groups_of_a_batch(precision, count, group, up):
    """50 x 50 cavities of one structure that end their solves at different passes, in groups
    with a remainder: bit for bit the problems alone (whose groups hold one), and within the
    solves' tolerance the stored operators."""
    from pycfd_b200.batch import BatchedSolver, BatchOptions
    re = np.geomspace(5.0, 3000.0, count)
    cfgs = [_cfg(50, 50, cases.bcs(top=("moving_wall", 0.3 + 0.01 * k)), re=float(re[k]), adaptive_dt=False, dt=1e-3,
                 t_end=10.0) for k in range(count)]

    def run(cfgs, **kw):
        b = BatchedSolver(cfgs, BatchOptions(precision=precision, inner_tol=1e-3, **kw))
        b.step(3)
        st = b.status()
        assert not st["status"].any() and not st["frozen"].any()
        return b, st["iterations"], [f.numpy() for f in b.fields]

    b, its, fields = run(cfgs)
    assert b.form() == {"pattern_structures": 1, "stored_structures": 0, "group": group, "up_group": up}
    assert len(set(its.tolist())) > 1
    some = sorted({0, 1, 2, group - 1, group, count // 2, count - 2, count - 1})
    for k in some:
        one, it1, f1 = run(cfgs[k:k + 1])
        assert one.form()["group"] == one.form()["up_group"] == 1
        assert it1[0] == its[k]
        for p, q in zip(fields[k], f1[0]):
            assert np.array_equal(p, q), k
    g, its_g, fields_g = run(cfgs, ell_group=1)
    assert g.form()["pattern_structures"] == 0
    assert np.abs(its - its_g).max() <= 3 * (4 if precision == "mixed" else 1)   # a pass or so per (inner) solve
    for x, y in zip(fields, fields_g):
        for p, q in zip(x, y):
            assert np.abs(p - q).max() <= 1e-8 * max(np.abs(f).max() for f in y)


def test_launch_counts_of_recorded_solves_beside_other_threads():
    """What a recording holds is counted apart from the launches that other threads make
    meanwhile: solves on four threads count what they count one after another."""
    import threading
    from pycfd_b200 import _lib
    L = _lib.load()
    sizes = [(64, 64), (96, 64), (80, 112), (128, 128)]
    rhs = [np.random.default_rng(k).standard_normal(n) for k, n in enumerate(sizes)]

    def work(k, s, barrier=None):
        with torch.cuda.stream(torch.cuda.Stream()):
            if barrier:
                barrier.wait()
            for _ in range(12):
                s.pressure_solver.solve(rhs[k])

    def total(threads):
        solvers = [_solver(_cfg(*n)) for n in sizes]
        torch.cuda.synchronize()
        n0 = L.pycfd_launch_count()
        if threads:
            b = threading.Barrier(len(sizes))
            ts = [threading.Thread(target=work, args=(k, s, b)) for k, s in enumerate(solvers)]
            [t.start() for t in ts]
            [t.join() for t in ts]
        else:
            [work(k, s) for k, s in enumerate(solvers)]
        assert all(s.form()["recorded_solves"] == 1 for s in solvers)
        return L.pycfd_launch_count() - n0

    one_by_one = total(False)
    assert one_by_one > 0 and total(True) == one_by_one


@pytest.mark.parametrize("field", ["a_indptr", "weighted_dinv", "p_indptr"])
def test_incomplete_levels_are_refused_whatever_the_form(field):
    """A level below the dense tail without its operator: read by no kernel of the pattern
    form, and refused by it as by the stored one."""
    import ctypes as C
    from pycfd_b200 import _lib
    from pycfd_b200.config import PressureSolver
    from pycfd_b200.solver import GpuOptions, native_desc
    L = _lib.load()
    s = _solver(_cfg(128, 128))
    assert s.form()["pattern_levels"] == 2 and len(s._levels) > 4
    for fused in (True, False):
        d, keep = native_desc(s.config, s.mesh, s.boundaries, s.solid, False, (), PressureSolver.MGCG,
                              GpuOptions(fused_restriction=fused), s._levels, s._cinv)
        e = d.levels[3]
        setattr(e, field, C.cast(C.c_void_p(0), type(getattr(e, field))))
        h = C.c_void_p()
        with pytest.raises(ValueError, match="level 3 lacks"):
            _lib.check(L.pycfd_solver_create(C.byref(d), C.byref(h)))


def test_wide_rows_keep_stored_operators():
    """Cells of aspect 2.2 and 1.5: rows of 349 and 576 entries above the closing level."""
    from pycfd_b200.batch import BatchedSolver, BatchOptions
    assert _solver(_cfg(192, 192, lx=2.2)).form()["pattern_levels"] > 0
    assert _solver(_cfg(192, 192, lx=1.5)).form()["pattern_levels"] == 0
    cfgs = [_cfg(96, 96, lx=lx, adaptive_dt=False, dt=1e-3, t_end=10.0) for lx in (1.0, 3.0, 2.2, 1.5)]
    b = BatchedSolver(cfgs, BatchOptions())
    assert (b.form()["pattern_structures"], b.form()["stored_structures"]) == (2, 2)
    g = BatchedSolver(cfgs, BatchOptions(ell_group=1))
    for x in (b, g):
        x.step(3)
        assert not x.status()["status"].any()
    for f, h in zip(b.fields, g.fields):
        for p, q in zip(f.numpy(), h.numpy()):
            assert np.abs(p - q).max() <= 1e-8 * max(np.abs(a).max() for a in h.numpy())
