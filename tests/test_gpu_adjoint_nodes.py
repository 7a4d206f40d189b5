"""The coordinate product's device helpers: vertices of elements, sums into nodes, the coordinates check."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["tri", "quad"])
@pytest.mark.parametrize("nx,nr", [(2, 1), (13, 7), (64, 33)])
def test_node_helpers_match_numpy(cuda, kind, nx, nr):
    """Exact: the sums are taken in np.add.at's order (vertices in turn, then elements)."""
    import torch

    cfg, mesh = pkg("config"), pkg("mesh")
    topo, xf, rf = mesh.channel_topology(kind, nx=nx, nr=nr)
    ops = pkg("operators").build_operators(topo, mesh.rectangle_coords(xf, rf), 1)
    m = pkg("adjoint").AdjointModel(ops, cfg.FlowConditions(), cfg.SolverOptions())
    rng = np.random.default_rng(1)
    gv = rng.standard_normal((2, m.NV, m.E))
    n = m.X0.shape[0]
    ref = np.zeros((n, 2))
    for c in range(2):
        np.add.at(ref[:, c], m.elem_nodes.T, gv[c])
    got = m._node_sums(torch.as_tensor(gv, device=m.device), n)
    assert np.array_equal(got.cpu().numpy(), ref)
    X = torch.as_tensor(rng.standard_normal((n, 2)), device=m.device)
    Xe = X.cpu().numpy()[m.elem_nodes]
    assert np.array_equal(m.verts(X).cpu().numpy(), np.concatenate([Xe[:, :, 0].T, Xe[:, :, 1].T]))
    with pytest.raises(IndexError):
        m.verts(X[:-1])
    # this model's own mesh for coordinates equal to the last bits, another one otherwise
    assert m.mesh_at(m.X0 * (1.0 + 2e-16)) is m.mesh
    assert m.mesh_at(m.X0 + 1e-9) is not m.mesh
    mesh_, pb = m._at(m.X0.clone(), torch.tensor(0.25, dtype=torch.float64, device=m.device))
    assert mesh_ is m.mesh and pb == 0.25
