"""The adjoint tile kernels on meshes of more blocks of 32 elements than CTAs fit the GPU (444 with stored
Jacobians), so that CTAs take several tiles, a partly filled last one among them, against the one-thread
kernel.  Tolerance as in test_gpu_tile.py: 100 terms x 1.3e-14."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg, rel
from test_gpu_tile import TOL, _states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nx,nr", [("quad", 160, 97), ("quad", 187, 161), ("tri", 160, 97)])
@pytest.mark.parametrize("p", [1, 2, 3])
def test_several_tiles_a_cta(cuda, kind, nx, nr, p, monkeypatch):
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
        march = ad.AdjointMarch(m, u, sd, 0.5)
        lam3, rel3, its, _ = march.solve(tolerance=0.0, max_iterations=3, check_interval=3)
        assert its == 3
        norm = float(march.t["res"].item())  # the defect of the run's last state
        out[name] = [m.vjp_state(u, la), m.adjoint_rate(u, la, sd), lam3.clone(), torch.tensor([rel3, norm])]
    for x, y in zip(out["t1"], out["split4"]):
        assert rel(y.cpu().numpy(), x.cpu().numpy()) < TOL
