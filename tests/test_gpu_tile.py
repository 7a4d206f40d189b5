"""The tile kernels (four lanes per element, FP64 tensor cores) at the edges of their tiling.

A warp owns eight elements, a block 32, and a CTA takes several blocks once the mesh has more than
fit the GPU at a time: meshes of a few elements, of one element more or less than a tile or a block,
and of more blocks than CTAs.  The reference is the one-thread kernel (held to the oracle elsewhere).

Tolerance: an output sums at most 32 point terms of at most 16-term interpolations, and the trace
tables differ between faces by up to 1.3e-14 (the reference's own round-off at cubic quadrilaterals),
so 100 terms x 1.3e-14 bounds the relative difference: 2e-12.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg, rel

pytestmark = pytest.mark.gpu
TOL = 2e-12

# (nx, nr) cells: triangles have twice as many elements, quadrilaterals as many
SIZES = [(2, 1), (3, 1), (4, 1), (5, 3), (8, 2), (11, 3), (33, 1), (160, 97)]


def _states(ops, seed):
    """Smooth flow with enough noise that some elements are limited and none is near vacuum."""
    rng = np.random.default_rng(seed)
    shape = (ops.n_elem, ops.ref.n_basis)
    rho = 1.0 + 0.2 * rng.uniform(-1, 1, shape)
    vx, vy, p = (rng.uniform(a, b, shape) for a, b in ((0.2, 0.9), (-0.3, 0.3), (0.4, 0.8)))
    return np.stack([rho, rho * vx, rho * vy, p / 0.4 + 0.5 * rho * (vx * vx + vy * vy)], -1)


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("nx,nr", SIZES)
def test_tiles_agree_with_one_thread(cuda, kind, p, nx, nr):
    cfg, mesh = pkg("config"), pkg("mesh")
    topo, xf, rf = mesh.channel_topology(kind, nx=nx, nr=nr)
    X = mesh.rectangle_coords(xf, rf)
    X = X + 0.1 / max(nx, nr) * np.sin(7.0 * X[:, ::-1])  # no two elements alike
    ops = pkg("operators").build_operators(topo, X, p, lean=True)
    U = _states(ops, 3)
    bk = pkg("backend").B200Backend(ops, cfg.FlowConditions(flux="hllc"), cfg.SolverOptions(cfl=0.5),
                                   device_metrics=True)
    out = {}
    for name in ("t1", "split4"):
        pkg("autotune").apply_variant(bk.mesh, name)
        R, wave = bk.residual(U)
        F, _ = bk.rate(U)
        U1, res, flags = bk.step_record(U)
        out[name] = (R, wave, F, U1, np.array([res])), flags
    for x, y in zip(out["t1"][0], out["split4"][0]):
        assert rel(y, x) < TOL
    assert np.array_equal(out["t1"][1], out["split4"][1])


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("nx,nr", SIZES)
def test_superbee_tiles_agree_with_one_thread(cuda, kind, p, nx, nr):
    """A step whose stages end with the slope limiter: state and residual.  The flags are not compared: an
    element with factor 1 counts as changed where ubar + (u - ubar) differs from u in the last bit, in
    the reference as here, so its flag depends on the average's rounding."""
    cfg, mesh = pkg("config"), pkg("mesh")
    topo, xf, rf = mesh.channel_topology(kind, nx=nx, nr=nr)
    X = mesh.rectangle_coords(xf, rf)
    X = X + 0.1 / max(nx, nr) * np.sin(7.0 * X[:, ::-1])
    ops = pkg("operators").build_operators(topo, X, p, lean=True)
    U = _states(ops, 6)
    bk = pkg("backend").B200Backend(ops, cfg.FlowConditions(flux="roe"),
                                    cfg.SolverOptions(cfl=0.5, limiter="superbee", tvb_constant=1.0), device_metrics=True)
    out = {}
    for name in ("t1", "split4"):
        pkg("autotune").apply_variant(bk.mesh, name)
        U1, res, _ = bk.step_record(U)
        out[name] = U1, np.array([res]), bk.limit(U)
    for x, y in zip(out["t1"], out["split4"]):
        assert rel(y, x) < TOL


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 2, 3])
def test_superbee_under_a_block_list(cuda, kind, p):
    """A stage that lists the first 128 elements only: the slope limiter still takes every element's
    average, from its own pass, as it does after the one-thread kernel with the same elements listed."""
    import ctypes as C

    import torch

    capi, cfg, mesh = pkg("capi"), pkg("config"), pkg("mesh")
    topo, xf, rf = mesh.channel_topology(kind, nx=33, nr=11)
    X = mesh.rectangle_coords(xf, rf)
    X = X + 0.003 * np.sin(7.0 * X[:, ::-1])
    ops = pkg("operators").build_operators(topo, X, p, lean=True)
    U = _states(ops, 7)
    bk = pkg("backend").B200Backend(ops, cfg.FlowConditions(flux="roe"),
                                   cfg.SolverOptions(cfl=0.5, limiter="superbee", tvb_constant=1.0), device_metrics=True)
    src = bk.mesh.pack(U, torch.empty(4 * bk.mesh.np_ * bk.mesh.E, dtype=torch.float64, device="cuda"))
    out = []
    for name in ("t1", "split4"):
        pkg("autotune").apply_variant(bk.mesh, name)
        mc = capi.Mesh()
        C.memmove(C.byref(mc), bk.mesh.c_ref, C.sizeof(capi.Mesh))
        listed = torch.arange(128 // int(bk.lib.nzb_block_width(C.byref(mc), 0)), dtype=torch.int32, device="cuda")
        mc.fwd_blocks, mc.n_fwd_blocks = listed.data_ptr(), listed.numel()
        bk.mesh.lim_means.fill_(1e3)
        new, dt = src.clone(), torch.ones(bk.mesh.E, dtype=torch.float64, device="cuda")
        a = capi.StageArgs()
        a.V, a.out, a.dt, a.dt_factor, a.a, a.b, a.stage = src.data_ptr(), new.data_ptr(), dt.data_ptr(), 0.1, 0.0, 1.0, 1
        capi.check(bk.lib.nzb_stage(C.byref(mc), bk._phys_ref, C.byref(a), bk._stream), "nzb_stage")
        out.append(new.cpu().numpy())
    assert rel(out[1], out[0]) < TOL


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("nx,nr", [s for s in SIZES if s != (160, 97)] + [(72, 100)])
def test_adjoint_tiles_agree_with_one_thread(cuda, kind, p, nx, nr, monkeypatch):
    """The product, the rate (both differentiate the fluxes in the kernel) and a run of three RK4 steps
    (stored face Jacobians) against the one-thread adjoint kernel."""
    import torch

    ad, cfg, mesh = pkg("adjoint"), pkg("config"), pkg("mesh")
    topo, xf, rf = mesh.channel_topology(kind, nx=nx, nr=nr)
    X = mesh.rectangle_coords(xf, rf)
    X = X + 0.1 / max(nx, nr) * np.sin(7.0 * X[:, ::-1])
    ops = pkg("operators").build_operators(topo, X, p)
    U = torch.as_tensor(_states(ops, 4), device="cuda")
    rng = np.random.default_rng(5)
    lam, seed = (torch.as_tensor(rng.standard_normal(tuple(U.shape)), device="cuda") for _ in range(2))
    out = {}
    for name in ("t1", "split4"):
        monkeypatch.setenv("NZB_VJP_VARIANT", name)
        m = ad.AdjointModel(ops, cfg.FlowConditions(flux="ausmup"), cfg.SolverOptions(cfl=0.5))
        u, la, sd = (ad.to_soa(x) for x in (U, lam, seed))
        am = ad.AdjointMarch(m, u, sd, 0.5)
        lam3, rel3, its, _ = am.solve(tolerance=0.0, max_iterations=3, check_interval=3)
        out[name] = [m.vjp_state(u, la), m.adjoint_rate(u, la, sd), lam3.clone(), torch.tensor([rel3])]
        assert its == 3
    for x, y in zip(out["t1"], out["split4"]):
        assert rel(y.cpu().numpy(), x.cpu().numpy()) < TOL


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 3])
def test_adjoint_march_with_any_workspace(cuda, kind, p, monkeypatch):
    """A run of RK4 steps with the caller's Jacobian workspace, with the march's own (the same bits) and
    with none (the products differentiate in place); the choice is made once."""
    import ctypes as C

    import torch

    ad, capi, cfg, mesh = pkg("adjoint"), pkg("capi"), pkg("config"), pkg("mesh")
    topo, xf, rf = mesh.channel_topology(kind, nx=11, nr=3)
    ops = pkg("operators").build_operators(topo, mesh.rectangle_coords(xf, rf), p)
    m = ad.AdjointModel(ops, cfg.FlowConditions(flux="ausmup"), cfg.SolverOptions(cfl=0.5))
    u = ad.to_soa(torch.as_tensor(_states(ops, 8), device="cuda"))
    sd = ad.to_soa(torch.as_tensor(np.random.default_rng(9).standard_normal((ops.n_elem, ops.ref.n_basis, 4)), device="cuda"))
    out = []
    for given in (True, False):
        if not given:
            monkeypatch.setattr(ad, "_jacobian_workspace", lambda *a: None)
        am = ad.AdjointMarch(m, u, sd, 0.5)
        out.append(am.solve(tolerance=0.0, max_iterations=3, check_interval=3)[0].clone())
        with pytest.raises(capi.NativeError, match="once"):
            capi.check(m.lib.nzb_adjoint_jacobians(am.handle, 0, None), "nzb_adjoint_jacobians")
    offs, h = np.zeros(1, np.int64), capi.P()
    capi.check(m.lib.nzb_adjoint_create(1, m.mesh.c_ref, C.byref(am.ph), C.byref(am.bf), offs.ctypes.data, C.byref(am.am),
                                        C.byref(h)), "nzb_adjoint_create")
    m.lib.nzb_adjoint_destroy(am.handle)
    am.handle = h.value
    own = am.solve(tolerance=0.0, max_iterations=3, check_interval=3)[0]
    assert torch.equal(own, out[0])
    assert rel(out[1].cpu().numpy(), out[0].cpu().numpy()) < TOL


@pytest.mark.parametrize("decade", [-30, -20, -10, -1, 0, 1, 10, 20, 29])
def test_reciprocals_are_accurate(cuda, decade):
    """1 / a and 1 / sqrt(a) of the fluxes against the division's and torch's.  The step's remainder is
    2^-60 relative; two roundings follow it in the reciprocal and three in the root (half a unit each, the
    first of them scaled by the small correction), and the compared values have half a unit themselves:
    at most two units in the last place."""
    import torch

    capi = pkg("capi")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(decade + 100)
    a = 10.0**decade * (1.0 + 9.0 * torch.rand(200_001, generator=gen, dtype=torch.float64, device="cuda"))
    r, q = torch.empty_like(a), torch.empty_like(a)
    capi.check(capi.load().nzb_reciprocals(a.data_ptr(), r.data_ptr(), q.data_ptr(), a.numel(),
                                           torch.cuda.current_stream().cuda_stream), "nzb_reciprocals")
    for got, ref in ((r, 1.0 / a), (q, 1.0 / torch.sqrt(a))):
        assert float(((got - ref).abs() / ref).max()) <= 2 * 2.0**-52


def test_a_lone_large_instance_keeps_the_one_thread_kernel():
    """Which buckets the exception to the variant table takes (autotune.bucket_context)."""
    at = pkg("autotune")
    assert at.bucket_context(1, at.LONE_ELEMENTS + 1, "batch") == "lone"
    assert at.bucket_context(1, at.LONE_ELEMENTS, "batch") == "batch"
    assert at.bucket_context(2, 10**6, "batch") == "batch"
    assert at.bucket_context(1, 10**6, "single") == "single"
    assert at.variant_for("tri", 3, "lone") == "t1"
