"""AdjointModel's own checks: what it builds at its first use and keeps is complete for callers on any
stream, and coordinates that do not cover the elements' nodes are refused before a kernel reads them."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg, rel

pytestmark = pytest.mark.gpu


def test_node_items_are_there_for_another_stream(cuda):
    """The first coordinate product on a busy stream, the second right after it on another one."""
    import torch

    cfg, mesh = pkg("config"), pkg("mesh")
    topo, xf, rf = mesh.channel_topology("quad", nx=64, nr=33)
    ops = pkg("operators").build_operators(topo, mesh.rectangle_coords(xf, rf), 1)
    m = pkg("adjoint").AdjointModel(ops, cfg.FlowConditions(), cfg.SolverOptions())
    gv = np.random.default_rng(1).standard_normal((2, m.NV, m.E))
    n = m.X0.shape[0]
    ref = np.zeros((n, 2))
    for c in range(2):
        np.add.at(ref[:, c], m.elem_nodes.T, gv[c])
    g = torch.as_tensor(gv, device=m.device)
    torch.cuda.synchronize()
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(20_000_000)  # some 10 ms
        first = m._node_sums(g, n)
    with torch.cuda.stream(other):
        second = m._node_sums(g, n)
    torch.cuda.synchronize()
    assert np.array_equal(first.cpu().numpy(), ref) and np.array_equal(second.cpu().numpy(), ref)


def test_short_coordinates_are_refused(cuda):
    import torch

    cfg, mesh, ad = pkg("config"), pkg("mesh"), pkg("adjoint")
    topo, xf, rf = mesh.channel_topology("tri", nx=5, nr=3)
    ops = pkg("operators").build_operators(topo, mesh.rectangle_coords(xf, rf), 1)
    m = ad.AdjointModel(ops, cfg.FlowConditions(), cfg.SolverOptions())
    U = torch.tensor([1.0, 0.5, 0.1, 2.0], dtype=torch.float64, device=m.device).repeat_interleave(m.NP * m.E)
    pb = torch.tensor(0.5, dtype=torch.float64, device=m.device)
    for X in (m.X0[:-1], m.X0[:, :1], m.X0.reshape(-1)):
        for call in (lambda: m.residual(U, X), lambda: m.vjp_state(U, U, X=X), lambda: m.vjp_coords(U, U, X),
                     lambda: ad.ResidualFunction(m, U, X, pb)):
            with pytest.raises(IndexError):
                call()
    longer = torch.cat([m.X0, m.X0[:1]])  # nodes that no element uses are allowed
    assert rel(m.residual(U, longer)[0].cpu(), m.residual(U)[0].cpu()) < 1e-12
    assert m.vjp_coords(U, U, longer)[0].shape == longer.shape
