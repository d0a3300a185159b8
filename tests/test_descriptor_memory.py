"""Host memory behind a native descriptor (no GPU needed): everything a descriptor points
at must be held by the list returned with it, since the hierarchy cache keeps only the
last few structures and a batch uploads after all its descriptors are made."""

import ctypes as C
import gc

import numpy as np
import pytest

import cases
from pycfd_b200.config import BCKind, BCSpec, PressureSolver, SimulationConfig
from pycfd_b200.hierarchy import assemble, build_hierarchy
from pycfd_b200.mesh import StructuredMesh
from pycfd_b200.solver import BoundaryInfo, GpuOptions, native_desc


def _held(keep, address, count, itemsize):
    """Whether an array of the list covers [address, address + count * itemsize)."""
    return any(isinstance(a, np.ndarray) and a.ctypes.data <= address
               and address + count * itemsize <= a.ctypes.data + a.nbytes for a in keep)


@pytest.mark.parametrize("nx,ny,fused", [(64, 64, True), (50, 40, False)])
def test_descriptor_holds_what_it_points_at(nx, ny, fused):
    cfg = cases.to_config(dict(nx=nx, ny=ny, re=100.0, pressure_solver="mgcg", boundary_config=cases.bcs()),
                          SimulationConfig, BCSpec, BCKind)
    mesh = StructuredMesh.from_config(cfg)
    bnd = BoundaryInfo(cfg.boundary_config, mesh)
    levels, cinv = build_hierarchy(assemble(nx, ny, mesh.dx, mesh.dy, False, False))
    d, keep = native_desc(cfg, mesh, bnd, np.zeros((nx, ny), bool), False, (), PressureSolver.MGCG,
                          GpuOptions(tail_ratio=16.0, fused_restriction=fused), levels, cinv)
    addr = lambda p: C.cast(p, C.c_void_p).value  # noqa: E731
    assert d.tail_level > 0
    n = levels[d.tail_level].n
    assert _held(keep, addr(d.tail_operator), n * n, 8)
    nc = levels[-1].n
    assert _held(keep, addr(d.coarsest_inverse), nc * nc, 8)
    for l, lv in enumerate(levels):
        e = d.levels[l]
        assert _held(keep, addr(e.weighted_dinv), lv.n, 8) and _held(keep, addr(e.active), lv.n, 1)
        for ptr, idx, val, on in ((e.a_indptr, e.a_indices, e.a_data, True), (e.p_indptr, e.p_indices, e.p_data, l > 0),
                                  (e.m_indptr, e.m_indices, e.m_data, fused and 1 <= l <= d.tail_level)):
            assert bool(ptr) == on
            if on:
                rows = levels[l - 1].n if ptr is e.p_indptr else lv.n
                assert _held(keep, addr(ptr), rows + 1, 8)
                assert _held(keep, addr(idx), ptr[rows], 4) and _held(keep, addr(val), ptr[rows], 8)
    # the values survive the hierarchy
    want = levels[d.tail_level].tails[cfg.mg_sweeps].copy()
    del levels, cinv, lv
    gc.collect()
    junk = [np.full(n * n, np.nan) for _ in range(8)]
    assert np.array_equal(np.ctypeslib.as_array(d.tail_operator, (n, n)), want)
    del junk
