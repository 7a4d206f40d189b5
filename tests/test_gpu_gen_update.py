"""nzb_gen_update, the stage update of the generic path as a call of its own, against its formulas in numpy."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,p,q,nx,nr", [("tri", 4, 1, 3, 1), ("quad", 1, 2, 13, 10), ("quad", 5, 1, 5, 3)])
def test_stage_updates(cuda, kind, p, q, nx, nr):
    """A handful of roundings an output (4 units in the last place of its largest term); the norm sums
    4 NP squares of up to 4 roundings a thread, then the block and the blocks: (4 NP + 40) x 1.1e-16 relative,
    all terms positive."""
    import torch

    capi, cfg = pkg("capi"), pkg("config")
    cs = pkg("nozzle").build_case(element=kind, order=p, nx=nx, nr=nr, geometry_order=q, area_ratio=2.0,
                                  flow=cfg.FlowConditions(flux="hllc"), options=cfg.SolverOptions(cfl=0.3))
    bk = pkg("backend").B200Backend(cs.operators, cs.flow, cs.options)
    E, NP = cs.operators.n_elem, cs.operators.ref.n_basis
    rng = np.random.default_rng(4)
    V, U0, F = (rng.standard_normal((E, NP, 4)) for _ in range(3))
    wave = rng.uniform(0.0, 2.0, E)
    wave[0] = 0.0  # floored
    dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    nb = int(bk.lib.nzb_gen_blocks(bk._gm))
    assert nb == -(-E // 128)
    t = {k: dev(v) for k, v in (("V", V), ("U0", U0), ("F", F), ("wave", wave))}
    dt, out = dev(np.zeros(E)), dev(np.zeros((E, NP, 4)))
    partial, res = dev(np.zeros(nb)), dev(np.zeros(1))
    area = bk._arr["elem_area"].cpu().numpy()
    w = np.array(list(bk.phys.norm_w))
    ref_dt = 0.2 * area / np.maximum(wave, 1e-10)
    for stage, a, b in ((1, 0.0, 1.0), (2, 0.75, 0.25), (3, 1.0 / 3.0, 2.0 / 3.0)):
        g = capi.GenUpdateArgs()
        g.stage, g.dt_factor, g.a, g.b = stage, 0.1, a, b
        g.V, g.F, g.wave, g.U0 = (t[k].data_ptr() for k in ("V", "F", "wave", "U0"))
        g.dt, g.out = dt.data_ptr(), out.data_ptr()
        g.partial = partial.data_ptr() if stage == 1 else None
        capi.check(bk.lib.nzb_gen_update(bk._gm, bk._phys_ref, C.byref(g), bk._stream), "nzb_gen_update")
        d = ref_dt[:, None, None]
        ref = a * U0 + b * (V + d * F)
        size = np.abs(a * U0) + np.abs(b * V) + np.abs(b * d * F)
        assert (np.abs(out.cpu().numpy() - ref) <= 4 * 2.3e-16 * size).all()
        assert (np.abs(dt.cpu().numpy() - ref_dt) <= 4 * 2.3e-16 * ref_dt).all()
    capi.check(bk.lib.nzb_norm_finalize(partial.data_ptr(), nb, 4.0 * E * NP, res.data_ptr(), bk._stream), "nzb_norm_finalize")
    want = np.sqrt(np.sum((F * w) ** 2) / (4.0 * E * NP))
    assert abs(float(res.item()) - want) <= (4 * NP + 40) * 1.1e-16 * want
