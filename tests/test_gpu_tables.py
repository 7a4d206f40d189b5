"""Quadrilateral tables with vertex functions other than the unit square's: the same elements with two of
their vertices listed in the other order.  The tile kernels do not take them, so split = 4 gives the
one-thread kernels' bits, which are those of the usual tables to round-off."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import pkg, rel
from test_gpu_lean_flux import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 2, 3])
def test_other_vertex_functions(cuda, p):
    import torch

    capi, cfg, layout, at = pkg("capi"), pkg("config"), pkg("layout"), pkg("autotune")
    lib = capi.load()
    ops, U = _case("quad", p)
    flow, opts = cfg.FlowConditions(flux="hllc"), cfg.SolverOptions()
    arrays = layout.host_arrays(ops)
    tables = layout.element_tables(ops.ref)
    nqv, npts = ops.ref.dgeom_dxi_vol.shape[1], ops.ref.n_basis
    swapped = dict(arrays)
    swapped["geo"] = np.ascontiguousarray(arrays["geo"][[0, 2, 1, 3, 4, 6, 5, 7]])
    # the slot: phi, w dphi (two), M^-1, the edge basis, its weights, mean and volume weights, then the vertices
    at_dgx = 3 * npts * nqv + npts * npts + (p + 1) * ops.ref.w_face.size + ops.ref.w_face.size + npts + nqv
    other = tables.copy()
    for k in range(2):
        lo = at_dgx + k * 4 * nqv
        other[lo:lo + 4 * nqv] = tables[lo:lo + 4 * nqv].reshape(4, nqv)[[0, 2, 1, 3]].ravel()
    assert np.array_equal(tables[at_dgx:at_dgx + 4 * nqv], np.asarray(ops.ref.dgeom_dxi_vol).ravel())
    ph = layout.physics_struct(flow, opts, ops.ref)
    lam = np.random.default_rng(7).standard_normal(U.shape)

    def results(arr, split):
        dm = layout.DeviceMesh(device=torch.device("cuda"), arrays=arr, ref=ops.ref)
        at.apply_variant(dm, "t1" if split == 1 else "split4")
        dm.vjp_split = split
        u, la = dm.pack(U, dm.state()), dm.pack(lam, dm.state())
        R, out = dm.state(), dm.state()
        capi.check(lib.nzb_residual(C.byref(dm.c), C.byref(ph), 0, u.data_ptr(), R.data_ptr(), None, dm.stream()), "nzb_residual")
        a = capi.AdjointArgs()
        a.mode, a.U, a.lam, a.out = capi.ADJ_VJP, u.data_ptr(), la.data_ptr(), out.data_ptr()
        capi.check(lib.nzb_vjp(C.byref(dm.c), C.byref(ph), C.byref(a), dm.stream()), "nzb_vjp")
        assert lib.nzb_block_width(C.byref(dm.c), 0) == lib.nzb_block_width(C.byref(dm.c), 1)
        return [x.cpu().numpy() for x in (R, out)]

    usual = results(arrays, 1)
    try:
        capi.check(lib.nzb_upload_tables(1, p, other.ctypes.data, other.size), "nzb_upload_tables")
        one, four = results(swapped, 1), results(swapped, 4)
    finally:
        capi.check(lib.nzb_upload_tables(1, p, tables.ctypes.data, tables.size), "nzb_upload_tables")
    for a, b, c in zip(usual, one, four):
        assert rel(b, a) < 2e-12 and np.array_equal(c, b)
    for a, b in zip(usual, results(arrays, 4)):
        assert rel(b, a) < 2e-12
