"""An adjoint march takes its Jacobian workspace with its first step."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


def test_no_workspace_for_a_defect_alone(cuda, monkeypatch):
    import torch

    ad, cfg, mesh = pkg("adjoint"), pkg("config"), pkg("mesh")
    topo, xf, rf = mesh.channel_topology("tri", nx=11, nr=3)
    ops = pkg("operators").build_operators(topo, mesh.rectangle_coords(xf, rf), 2)
    monkeypatch.setenv("NZB_VJP_VARIANT", "split4")
    m = ad.AdjointModel(ops, cfg.FlowConditions(), cfg.SolverOptions(cfl=0.2))
    taken = []
    take = ad._jacobian_workspace
    monkeypatch.setattr(ad, "_jacobian_workspace", lambda *a: taken.append(take(*a)) or taken[-1])
    U = torch.tensor([1.0, 0.5, 0.1, 2.0], dtype=torch.float64, device=m.device).repeat_interleave(m.NP * m.E)
    zero = ad.AdjointMarch(m, U, torch.zeros_like(U), 0.2)
    assert zero.solve(max_iterations=4)[2:] == (0, True) and not taken
    seed = torch.as_tensor(np.random.default_rng(1).standard_normal(U.numel()), device=m.device)
    march = ad.AdjointMarch(m, U, seed, 0.2)
    for _ in range(2):
        assert march.solve(tolerance=0.0, max_iterations=4, check_interval=2)[2] == 4
    assert len(taken) == 1 and taken[0] is not None
