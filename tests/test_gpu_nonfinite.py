"""An infinite or NaN energy at one corner of an element: which elements' results it reaches, in the tile, the
adjoint tile and the generic kernels.  Only the element itself and its face neighbours read it, and the tile
kernel's results are non-finite where the one-thread kernel's are: an infinite energy gives an infinite
wave speed (the local step it bounds is zero)."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg, rel
from test_gpu_lean_flux import _backend, _case

pytestmark = pytest.mark.gpu


def _reached(ops, e):
    """e and its face neighbours, e an element without a boundary face."""
    pairs = np.asarray(ops.topology.edges.iedge_elem)
    near = {int(x) for pair in pairs if e in pair for x in pair}
    assert len(near) == 1 + (3 if ops.ref.kind == "tri" else 4)
    out = np.zeros(ops.n_elem, bool)
    out[list(near)] = True
    return out


def _interior(ops):
    pairs = np.asarray(ops.topology.edges.iedge_elem)
    count = np.bincount(pairs.ravel(), minlength=ops.n_elem)
    return int(np.flatnonzero(count == (3 if ops.ref.kind == "tri" else 4))[0])


def _ok(x):
    return np.isfinite(x).reshape(len(x), -1).all(1)


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("flux", ["roe", "hllc", "ausmup"])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_the_element_kernels(cuda, kind, p, flux, bad):
    ops, U = _case(kind, p)
    bk = _backend(ops, flux)
    R0, w0 = bk.residual(U)
    e = _interior(ops)
    U[e, 0, 3] = bad
    near = _reached(ops, e)
    out = {}
    for name in ("t1", "split4"):
        pkg("autotune").apply_variant(bk.mesh, name)
        R, wave = bk.residual(U)
        F, _ = bk.rate(U)
        assert not _ok(R)[e] and _ok(R)[~near].all()
        assert rel(R[~near], R0[~near]) < 2e-12 and rel(wave[~near], w0[~near]) < 2e-12
        out[name] = _ok(R), _ok(F), np.isposinf(wave)
        assert not np.isfinite(bk.step_record(U)[1])
    assert out["t1"][2].any() == (bad == np.inf)
    for x, y in zip(out["t1"], out["split4"]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("kind,p,q", [("tri", 4, 1), ("tri", 2, 2), ("quad", 2, 2), ("quad", 4, 1)])
@pytest.mark.parametrize("flux", ["roe", "hllc", "ausmup"])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_the_generic_kernels(cuda, kind, p, q, flux, bad):
    cfg = pkg("config")
    cs = pkg("nozzle").build_case(element=kind, order=p, nx=7, nr=3, geometry_order=q, area_ratio=2.0,
                                  flow=cfg.FlowConditions(flux=flux), options=cfg.SolverOptions(cfl=0.3))
    bk = pkg("backend").B200Backend(cs.operators, cs.flow, cs.options)
    assert type(bk).__name__ == "GenericB200Backend"
    U = np.array(cs.initial_state())
    R0, w0 = bk.residual(U)
    e = _interior(cs.operators)
    U[e, 0, 3] = bad
    near = _reached(cs.operators, e)
    R, wave = bk.residual(U)
    assert not _ok(R)[e] and _ok(R)[~near].all()
    assert rel(R[~near], R0[~near]) < 2e-12 and rel(wave[~near], w0[~near]) < 2e-12
    if bad == np.inf:
        assert np.isposinf(wave[e])
    assert not np.isfinite(bk.run(U, 1, "ssprk3")[1])


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("where", ["state", "lambda"])
def test_the_adjoint_kernels(cuda, kind, p, bad, where, monkeypatch):
    """The product (fluxes differentiated in place) and a run of two steps (stored Jacobians): what a bad
    element reaches is at most its face neighbours a product, and the other elements keep their values."""
    import torch

    ad, cfg = pkg("adjoint"), pkg("config")
    ops, U = _case(kind, p)
    rng = np.random.default_rng(5)
    lam, seed = (rng.standard_normal(U.shape) for _ in range(2))
    e = _interior(ops)
    near = _reached(ops, e)
    clean = U.copy()
    (U if where == "state" else lam)[e, 0, 3] = bad
    soa = lambda x: ad.to_soa(torch.as_tensor(x, device="cuda"))  # noqa: E731
    for name in ("t1", "split4"):
        monkeypatch.setenv("NZB_VJP_VARIANT", name)
        m = ad.AdjointModel(ops, cfg.FlowConditions(flux="ausmup"), cfg.SolverOptions(cfl=0.2))
        lam0 = np.where(np.isfinite(lam), lam, 0.0)
        want = ad.from_soa(m.vjp_state(soa(clean), soa(lam0)), m.E, m.NP).cpu().numpy()
        got = ad.from_soa(m.vjp_state(soa(U), soa(lam)), m.E, m.NP).cpu().numpy()
        assert not _ok(got)[e] and _ok(got)[~near].all()
        assert rel(got[~near], want[~near]) < 2e-12
        seed_bad = seed.copy()
        if where == "lambda":
            seed_bad[e, 0, 3] = bad
        march = ad.AdjointMarch(m, soa(U if where == "state" else clean), soa(seed_bad), 0.2)
        lam1, _, its, converged = march.solve(tolerance=0.0, max_iterations=1, check_interval=1)
        assert not converged
        # four stages: the elements four faces and more away are untouched
        far = ~near
        pairs = np.asarray(ops.topology.edges.iedge_elem)
        for _ in range(3):
            grow = ~far
            for a, b in pairs:
                if not far[a] or not far[b]:
                    grow[a] = grow[b] = True
            far = ~grow
        x = ad.from_soa(lam1, m.E, m.NP).cpu().numpy()
        assert far.any() and _ok(x)[far].all()
