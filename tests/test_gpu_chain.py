"""Chained launches (each kernel of a march starts while the one before it drains) against the same work
launched apart, where no two kernels are resident together: the same kernels on the same data, so the same
bits.  Sizes: a few elements, and up to one full wave of CTAs (444 blocks of 32 elements), where launches
are chained and neighbouring CTAs share cache lines from different SMs; element counts that are no multiple
of a cache line's 16 doubles; past one wave, where the larger kernels' launches are not chained."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu
SIZES = [(11, 3), (67, 71), (117, 59), (97, 97)]
STEPS = 5


def _ops(kind, p, nx, nr):
    mesh = pkg("mesh")
    topo, xf, rf = mesh.channel_topology(kind, nx=nx, nr=nr)
    X = mesh.rectangle_coords(xf, rf)
    return pkg("operators").build_operators(topo, X + 0.1 / max(nx, nr) * np.sin(7.0 * X[:, ::-1]), p, lean=True)


def _states(ops, seed):
    rng = np.random.default_rng(seed)
    shape = (ops.n_elem, ops.ref.n_basis)
    rho = 1.0 + 0.2 * rng.uniform(-1, 1, shape)
    vx, vy, p = (rng.uniform(a, b, shape) for a, b in ((0.2, 0.9), (-0.3, 0.3), (0.4, 0.8)))
    return np.stack([rho, rho * vx, rho * vy, p / 0.4 + 0.5 * rho * (vx * vx + vy * vy)], -1)


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("limiter", ["positivity", "superbee"])
@pytest.mark.parametrize("nx,nr", SIZES)
def test_a_march_is_its_steps(cuda, kind, p, limiter, nx, nr):
    """run(n) against n times step_record, whose stages are separate, unchained launches."""
    cfg = pkg("config")
    ops = _ops(kind, p, nx, nr)
    U = _states(ops, 11)
    bk = pkg("backend").B200Backend(ops, cfg.FlowConditions(flux="hllc"),
                                    cfg.SolverOptions(cfl=0.2, limiter=limiter, tvb_constant=1.0), device_metrics=True)
    for scheme in ("ssprk3", "euler"):
        V, res = U, 0.0
        for _ in range(STEPS):
            V, res, _ = bk.step_record(V, scheme)
        W, res_run = bk.run(U, STEPS, scheme)
        assert np.isfinite(V).all()
        assert np.array_equal(W, V) and res_run == res


@pytest.mark.parametrize("kind,p,q", [("tri", 4, 1), ("tri", 2, 2), ("quad", 2, 2)])
@pytest.mark.parametrize("limiter", ["positivity", "superbee"])
@pytest.mark.parametrize("nx,nr", [(5, 3), (37, 31)])
def test_a_generic_march_is_its_steps(cuda, kind, p, q, limiter, nx, nr):
    """run(n) against n calls of run(1): the first launch of a call is not chained."""
    cfg = pkg("config")
    cs = pkg("nozzle").build_case(element=kind, order=p, nx=nx, nr=nr, geometry_order=q, area_ratio=2.0,
                                  flow=cfg.FlowConditions(flux="hllc"), options=cfg.SolverOptions(cfl=0.2, limiter=limiter))
    bk = pkg("backend").B200Backend(cs.operators, cs.flow, cs.options)
    U = cs.initial_state()
    for scheme in ("ssprk3", "euler"):
        V, res = U, 0.0
        for _ in range(STEPS):
            V, res = bk.run(V, 1, scheme)
        W, res_run = bk.run(U, STEPS, scheme)
        assert np.array_equal(W, V) and res_run == res


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("nx,nr", SIZES)
def test_an_adjoint_march_is_its_steps(cuda, kind, p, nx, nr):
    """A run of n RK4 steps against n runs of one: the first launch of a run is not chained."""
    import torch

    ad, cfg = pkg("adjoint"), pkg("config")
    ops = _ops(kind, p, nx, nr)
    if kind == "quad":
        ops = pkg("operators").build_operators(ops.topology, ops.node_coords, p)
    m = ad.AdjointModel(ops, cfg.FlowConditions(flux="hllc"), cfg.SolverOptions(cfl=0.2))
    u = ad.to_soa(torch.as_tensor(_states(ops, 12), device="cuda"))
    seed = ad.to_soa(torch.as_tensor(np.random.default_rng(13).standard_normal((ops.n_elem, ops.ref.n_basis, 4)),
                                     device="cuda"))
    out = []
    for interval in (STEPS, 1):
        am = ad.AdjointMarch(m, u, seed, 0.2)
        lam, rel, its, _ = am.solve(tolerance=0.0, max_iterations=STEPS, check_interval=interval)
        out.append((lam.clone(), rel, its))
    assert torch.isfinite(out[0][0]).all()
    assert torch.equal(out[0][0], out[1][0]) and out[0][1:] == out[1][1:]


@pytest.mark.parametrize("limiter", ["positivity", "superbee"])
def test_a_batch_march_is_its_steps(cuda, limiter):
    """Chunks of n steps against chunks of one, several instances of each element type: meshes of six
    and four elements, so that a warp's tile holds parts of two, and a larger one."""
    cfg, batch = pkg("config"), pkg("batch")
    out = []
    for interval in (10, 1):
        opts = cfg.SolverOptions(cfl=0.2, limiter=limiter, tvb_constant=1.0, tolerance=1e-30, max_iterations=11,
                                 check_interval=interval, print_interval=0)
        insts = []
        for kind in ("tri", "quad"):
            for p in (1, 2, 3):
                for nx, nr in ((3, 1), (2, 1), (41, 23), (3, 1)):
                    ops = _ops(kind, p, nx, nr)
                    insts.append(batch.Instance(ops, cfg.FlowConditions(flux="hllc"), opts, _states(ops, 14)))
        solver = batch.BatchSolver(insts)
        solver.run()
        out.append(solver.results())
    for a, b in zip(*out):
        assert a.iterations == b.iterations == 11 and a.residual == b.residual
        assert np.array_equal(a.U, b.U)
