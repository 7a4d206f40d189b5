"""The Superbee limiter in a batch of more blocks than CTAs fit the GPU, with several instances: a CTA takes
tiles of different instances, a warp's tile parts of two, and each instance's maxima are its own.  One step of
the tile kernels against the one-thread kernels; tolerance as in test_gpu_tile.py (100 terms x 1.3e-14)."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg, rel
from test_gpu_tile import TOL, _states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,sizes", [("tri", [(3, 1), (67, 71), (2, 1), (97, 59), (5, 1)]),
                                        ("quad", [(3, 1), (89, 101), (5, 1), (97, 83), (7, 1)])])
@pytest.mark.parametrize("p", [1, 2, 3])
def test_maxima_are_an_instances_own(cuda, kind, sizes, p, monkeypatch):
    cfg, mesh, batch = pkg("config"), pkg("mesh"), pkg("batch")
    opts = cfg.SolverOptions(cfl=0.3, limiter="superbee", tvb_constant=1.0, tolerance=1e-30, max_iterations=1,
                             check_interval=1, print_interval=0)
    insts = []
    for k, (nx, nr) in enumerate(sizes):
        topo, xf, rf = mesh.channel_topology(kind, nx=nx, nr=nr)
        X = mesh.rectangle_coords(xf, rf)
        ops = pkg("operators").build_operators(topo, X + 0.1 / max(nx, nr) * np.sin(7.0 * X[:, ::-1]), p, lean=True)
        U = _states(ops, 20 + k) * 2.0**k  # maxima that differ from instance to instance
        insts.append(batch.Instance(ops, cfg.FlowConditions(flux="roe"), opts, U))
    assert sum(i.ops.n_elem for i in insts) > 444 * 32
    out = {}
    for name in ("t1", "split4"):
        monkeypatch.setenv("NZB_VARIANT", name)
        solver = batch.BatchSolver(insts)
        solver.run()
        out[name] = solver.results()
    for a, b in zip(out["t1"], out["split4"]):
        assert a.iterations == b.iterations == 1
        assert rel(b.U, a.U) < TOL and abs(b.residual - a.residual) < TOL * a.residual
