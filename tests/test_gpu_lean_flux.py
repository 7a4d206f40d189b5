"""The short reciprocals and roots of the tile and generic kernels' fluxes, and the states at which the
fluxes' intermediate products must not overflow."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg, rel

pytestmark = pytest.mark.gpu


def _case(kind, p, nx=11, nr=3):
    mesh = pkg("mesh")
    topo, xf, rf = mesh.channel_topology(kind, nx=nx, nr=nr)
    X = mesh.rectangle_coords(xf, rf)
    ops = pkg("operators").build_operators(topo, X + 0.01 * np.sin(7.0 * X[:, ::-1]), p)
    rng = np.random.default_rng(3)
    shape = (ops.n_elem, ops.ref.n_basis)
    rho = 1.0 + 0.2 * rng.uniform(-1, 1, shape)
    vx, vy, pr = (rng.uniform(a, b, shape) for a, b in ((0.2, 0.9), (-0.3, 0.3), (0.4, 0.8)))
    return ops, np.stack([rho, rho * vx, rho * vy, pr / 0.4 + 0.5 * rho * (vx * vx + vy * vy)], -1)


def _backend(ops, flux, **kw):
    cfg = pkg("config")
    return pkg("backend").B200Backend(ops, cfg.FlowConditions(flux=flux, **kw), cfg.SolverOptions(cfl=0.2))


@pytest.mark.parametrize("decade", [-30, -20, -10, -1, 0, 1, 10, 20, 29])
def test_roots_are_rounded_once(cuda, decade):
    """The root's remainder is 2^-59 of it before its one rounding: at most one unit in the last place from
    the correctly rounded one, and different from it at all for about one argument in 2^-59 / 2^-54 = 32."""
    import torch

    capi = pkg("capi")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(decade + 200)
    a = 10.0**decade * (1.0 + 9.0 * torch.rand(200_001, generator=gen, dtype=torch.float64, device="cuda"))
    s = torch.empty_like(a)
    capi.check(capi.load().nzb_roots(a.data_ptr(), s.data_ptr(), a.numel(), torch.cuda.current_stream().cuda_stream),
               "nzb_roots")
    off = (s.view(torch.int64) - torch.sqrt(a).view(torch.int64)).abs()
    assert int(off.max()) <= 1 and float((off > 0).double().mean()) < 1.0 / 32


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("flux", ["roe", "hllc", "ausmup"])
def test_large_densities(cuda, kind, p, flux):
    """A state times 2^520: a product of two densities overflows, nothing the interface fluxes need does.  The
    tile kernel against the one-thread kernel, as at ordinary states (100 terms x 1.3e-14, test_gpu_tile.py),
    on the elements without a boundary face: a boundary's total pressure does not scale along, so the speeds
    there are differences of numbers 150 decades apart."""
    ops, U = _case(kind, p)
    inner = np.bincount(np.asarray(ops.topology.edges.iedge_elem).ravel(), minlength=ops.n_elem) == (3 if kind == "tri" else 4)
    U = U * 2.0**520
    bk = _backend(ops, flux)
    out = {}
    for name in ("t1", "split4"):
        pkg("autotune").apply_variant(bk.mesh, name)
        out[name] = [bk.residual(U)[0] * 2.0**-520, bk.residual(U)[1], bk.rate(U)[0] * 2.0**-520]
    for x, y in zip(out["t1"], out["split4"]):
        assert np.isfinite(x).all() and np.isfinite(y).all() and rel(y[inner], x[inner]) < 2e-12


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("flux", ["hllc"])
@pytest.mark.parametrize("low_mach", [0.05, 0.4, 5.0])
def test_low_mach_hllc(cuda, kind, p, flux, low_mach):
    """HLLC with the low-Mach scaling of its wave speeds below, across and above the states' Mach numbers."""
    ops, U = _case(kind, p)
    bk = _backend(ops, flux, hllc_low_mach=low_mach)
    out = {}
    for name in ("t1", "split4"):
        pkg("autotune").apply_variant(bk.mesh, name)
        out[name] = [*bk.residual(U), bk.rate(U)[0]]
    for x, y in zip(out["t1"], out["split4"]):
        assert rel(y, x) < 2e-12
