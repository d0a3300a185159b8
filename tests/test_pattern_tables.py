"""Tables of row patterns against the products they hold (no GPU needed).

The library's own host code builds the tables of a hierarchy and walks them entry by
entry as the kernels do; the walk must give M b, and Q x + G b, of every level in both
storage types.  Bent channels are the masks where a coarse level's rows take the widths
(6 and 5 entries) of the usual level-0 product.
"""

import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import cases
import native_build
from pycfd_b200.config import BCKind, BCSpec, PressureSolver, SimulationConfig
from pycfd_b200.hierarchy import hierarchy_for, tail_level
from pycfd_b200.mesh import StructuredMesh
from pycfd_b200.solver import BoundaryInfo, GpuOptions, native_desc


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    L = native_build.load("pattern_tables", tmp_path_factory.mktemp("native"))
    L.pt_build.restype = C.c_void_p
    L.pt_build.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p]
    L.pt_free.argtypes = [C.c_void_p]
    L.pt_ok.argtypes = [C.c_void_p, C.c_int]
    L.pt_info.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.POINTER(C.c_int)]
    L.pt_apply.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    return L


def channel(nx, ny, w, i, j):
    """All solid but an L-shaped channel of width w with its corner at (i, j)."""
    solid = np.ones((nx, ny), bool)
    solid[i:i + w, j:] = False
    solid[i:, j:j + w] = False
    return solid


def circle(nx, ny):
    x, y = np.meshgrid(np.arange(nx) + 0.5, np.arange(ny) + 0.5, indexing="ij")
    return (x - 0.4 * nx) ** 2 + (y - 0.5 * ny) ** 2 < (0.2 * min(nx, ny)) ** 2


def problem(nx, ny, solid, ratio, bc=None, aspect=1.0):
    """(levels, closing level, descriptor, what it points to, solvable cells)."""
    cfg = cases.to_config(dict(nx=nx, ny=ny, lx=aspect * nx / 64.0, ly=ny / 64.0, re=100.0,
                               pressure_solver="mgcg",
                               boundary_config=bc or cases.bcs()), SimulationConfig, BCSpec, BCKind)
    mesh = StructuredMesh.from_config(cfg)
    bnd = BoundaryInfo(cfg.boundary_config, mesh)
    op, (levels, cinv) = hierarchy_for(nx, ny, mesh.dx, mesh.dy, bnd.periodic_x, bnd.periodic_y, solid,
                                       bnd.dirichlet_pressure() or None)
    body = np.zeros((nx, ny), bool) if solid is None else solid
    d, keep = native_desc(cfg, mesh, bnd, body, solid is not None, (), PressureSolver.MGCG,
                          GpuOptions(tail_ratio=ratio), levels, cinv)
    t = tail_level(levels, ratio) or len(levels) - 1
    return levels, t, d, keep, np.asarray(op.fluid, np.uint8).ravel()


def products(levels, l):
    """M of level l + 1 and (Q, G) of level l, in double."""
    f, P = levels[l], levels[l + 1].P.tocsr()
    A, W = f.A.tocsr(), sp.diags(np.asarray(f.weighted_dinv))
    eye = sp.identity(f.n, format="csr")
    return P.T @ (eye - A @ W), (eye - W @ A) @ P, W @ (2.0 * eye - A @ W)


CHANNELS = [(135, 145, 1, 3, 6, None), (151, 177, 1, 111, 110, None), (51, 71, 1, 14, 23, 16.0),
            (13, 78, 1, 10, 0, 16.0)]


def check(L, nx, ny, solid, ratio, bc=None):
    levels, t, d, keep, solvable = problem(nx, ny, solid, ratio, bc)
    rng = np.random.default_rng(nx * 1000 + ny)
    h = L.pt_build(C.cast(d.levels, C.c_void_p), t, 1, solvable.ctypes.data)
    raw = set()   # (level, widest row of Q, of G) as the products have them
    try:
        for single in (0, 1):
            assert L.pt_ok(h, single)
            # FP32 entries are rounded once; the products and sums of the walk are double
            tol = 1e-6 if single else 1e-14
            for l in range(t):
                M, Q, G = products(levels, l)
                live = solvable.astype(float) if l == 0 else np.ones(levels[l].n)
                b = rng.standard_normal(levels[l].n) * live   # the projected residual is zero on solid cells
                x = rng.standard_normal(levels[l + 1].n)
                for up, want, parts, s1 in ((0, M @ b, (1, 2, 3, 8), b), (1, Q @ x + G @ b, (1, 2, 3, 8), x)):
                    info = (C.c_int * 5)()
                    L.pt_info(h, single, l if up else l + 1, up, info)
                    if not (up and l == 0):
                        assert info[4] == 0 and info[0] % 4 == 0 and info[1] % 4 == 0
                    if up and not single:
                        Gl = (G @ sp.diags(live)).tocsr()
                        Gl.eliminate_zeros()
                        raw.add((l, int(np.diff(Q.tocsr().indptr).max()), int(np.diff(Gl.indptr).max())))
                    for p in parts if not (up and l == 0) else (1,):
                        y = np.empty(len(want))
                        L.pt_apply(h, single, l if up else l + 1, up, p, s1.ctypes.data, b.ctypes.data, y.ctypes.data)
                        # a row adds at most a few hundred products of this size
                        size = max(np.abs(want).max(), np.abs(s1).max(), np.abs(b).max())
                        assert np.abs(y - want).max() <= tol * 100 * size, (single, l, up, p)
    finally:
        L.pt_free(h)
    return raw


@pytest.mark.parametrize("nx,ny,w,i,j,ratio", CHANNELS)
def test_tables_of_bent_channels(lib, nx, ny, w, i, j, ratio):
    raw = check(lib, nx, ny, channel(nx, ny, w, i, j), ratio)
    assert any(l >= 1 and q == 6 and g == 5 for l, q, g in raw), raw   # the mask still has that coarse level


@pytest.mark.parametrize("nx,ny,solid,ratio,bc", [
    (64, 64, False, None, None), (97, 61, True, 16.0, None), (96, 130, True, 16.0, cases.PER),
    (150, 61, True, None, cases.bcs(right=("pressure_outlet", 0.0, "uniform", 0.3))), (40, 6, False, 16.0, None)])
def test_tables_of_open_grids(lib, nx, ny, solid, ratio, bc):
    check(lib, nx, ny, circle(nx, ny) if solid else None, ratio, bc)


def pegs(n, seed=0):
    """One solid cell at a random place of every 4 x 4 block: nearly every coarse row differs."""
    rng = np.random.default_rng(seed)
    solid = np.zeros((n, n), bool)
    for a in range(0, n - 3, 4):
        for b in range(0, n - 3, 4):
            solid[a + rng.integers(3), b + rng.integers(3)] = True
    return solid


def test_tables_of_a_mask_with_a_pattern_per_row(lib):
    check(lib, 96, 96, pegs(96), 16.0)


@pytest.mark.parametrize("n,alone,batch", [(256, True, True), (272, False, True), (560, False, False)])
def test_how_many_patterns_are_taken(lib, n, alone, batch):
    """Level 1 has 16384 rows at 256 x 256 (no limit below), 18496 at 272 x 272 (a single
    problem keeps its stored operators), 78400 at 560 x 560 (more than a row can name)."""
    levels, t, d, keep, solvable = problem(n, n, pegs(n), 16.0)
    for any_, want in ((0, alone), (1, batch)):
        h = lib.pt_build(C.cast(d.levels, C.c_void_p), t, any_, solvable.ctypes.data)
        assert bool(lib.pt_ok(h, 0)) == bool(lib.pt_ok(h, 1)) == want
        lib.pt_free(h)


@pytest.mark.parametrize("nx", [1, 2, 3, 31, 1000])
@pytest.mark.parametrize("ny", [1, 2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 64, 100])
@pytest.mark.parametrize("K", [4, 24, 60, 400])
def test_tiles_cover_every_row_once(lib, nx, ny, K):
    """The rows a launch's threads take, each by as many parts as the row has."""
    out = (C.c_int * (nx * ny))()
    parts = lib.pt_cover(nx, ny, K, out)
    assert parts >= 1 and all(v == parts for v in out)


@pytest.mark.parametrize("nx,ny,fits", [(524280, 17, True), (524281, 17, False), (2, 524281, True), (600000, 4, True),
                                        (1048560, 16, True), (1048561, 16, False), (8192, 8192, True),
                                        (20000, 1, True)])
def test_grids_of_the_products(lib, nx, ny, fits):
    """A tile is 8 rows along x by 32 along y, 16 by 16 on a grid no wider than that: more
    than 65,535 tiles along x are not launched."""
    assert bool(lib.pt_fits(nx, ny, 24)) == fits


@pytest.mark.parametrize("nx,ny,aspect,ratio,width,alone,batch", [
    (96, 96, 1.0, 16.0, 37, True, True), (96, 96, 3.0, 16.0, 225, True, True), (96, 96, 2.2, 16.0, 349, True, False),
    (96, 96, 6.0, 16.0, 425, False, False), (96, 96, 1.5, 16.0, 576, False, False),
    (128, 128, 2.0, None, 79, True, True)])
def test_wide_rows_keep_stored_operators(lib, nx, ny, aspect, ratio, width, alone, batch):
    """Anisotropic cells: the widest row of A on a level above the closing one decides,
    at 400 entries for a problem alone and at 256 in a batch."""
    levels, t, d, keep, solvable = problem(nx, ny, None, ratio, aspect=aspect)
    widest = max(int(np.diff(lv.A.tocsr().indptr).max()) for lv in levels[:t])
    assert widest == width
    for b, want in ((0, alone), (1, batch)):
        h = lib.pt_build(C.cast(d.levels, C.c_void_p), t, b, solvable.ctypes.data)
        assert bool(lib.pt_ok(h, 0)) == bool(lib.pt_ok(h, 1)) == want
        lib.pt_free(h)
