"""Large arbitrary states in a batch: their bits are theirs alone, and nozzles of any size follow the table."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


def _instance(kind, p, nx, nr, seed):
    cfg, mesh, batch = pkg("config"), pkg("mesh"), pkg("batch")
    topo, xf, rf = mesh.channel_topology(kind, nx=nx, nr=nr)
    ops = pkg("operators").build_operators(topo, mesh.rectangle_coords(xf, rf), p, lean=True)
    opts = cfg.SolverOptions(cfl=0.2, tolerance=1e-30, max_iterations=5, check_interval=2, print_interval=0)
    return batch.Instance(ops, cfg.FlowConditions(flux="hllc"), opts,
                          pkg("autotune").random_states(ops.n_elem, ops.ref.n_basis, seed=seed))


@pytest.mark.parametrize("kind,nx,nr", [("tri", 150, 57), ("quad", 167, 101)])
def test_a_large_state_has_the_same_bits_alone_and_beside_others(cuda, kind, nx, nr):
    large, other, small = (_instance(kind, 2, a, b, s) for a, b, s in ((nx, nr, 1), (nx, nr, 2), (11, 3, 3)))
    out = []
    for members in ([large], [large, other], [small, other, large]):
        solver = pkg("batch").BatchSolver(members)
        solver.run()
        at = [i for i, m in enumerate(members) if m is large][0]
        out.append(solver.results()[at])
    for r in out[1:]:
        assert r.iterations == out[0].iterations and r.residual == out[0].residual
        assert np.array_equal(r.U, out[0].U, equal_nan=True)


def test_a_large_nozzle_follows_the_table(cuda):
    cfg, batch, at = pkg("config"), pkg("batch"), pkg("autotune")
    cs = pkg("nozzle").build_case(element="tri", order=1, refine=0, nx=150, nr=57, area_ratio=2.0, lean=True,
                                  flow=cfg.FlowConditions(flux="hllc"), options=cfg.SolverOptions(max_iterations=2))
    assert cs.operators.n_elem > at.LONE_ELEMENTS
    nozzle = batch.Instance(cs.operators, cs.flow, cs.options, None, cs.geometry.length, cs.geometry)
    solver = batch.BatchSolver([nozzle])
    assert solver.meshes[0].split == at.VARIANTS[at.variant_for("tri", 1, "batch")]["split"]
