"""The warp-per-element generic kernels over their node tiles and element remainders, against the oracle.

One to five tiles of eight nodes (3 to 36 basis functions), element counts that leave a block of four
warps partly filled, straight and curved.  Tolerance: the folded operators carry M^-1, whose condition
number reaches 1e4 at order 7, and an output sums at most 150 terms: 1e4 x 150 x 1.1e-16 = 2e-10 for
rates and steps; the unfolded residual has no inverse mass, 150 x 1e-14 (basis tables) = 2e-12.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import pkg, rel
from oracle import dg_oracle as orc

pytestmark = pytest.mark.gpu

CASES = [("tri", 1, 2), ("tri", 3, 2), ("tri", 4, 1), ("tri", 5, 1), ("tri", 6, 1), ("tri", 7, 1),
         ("quad", 1, 2), ("quad", 2, 2), ("quad", 4, 1), ("quad", 5, 1)]


@pytest.mark.parametrize("kind,p,q", CASES)
@pytest.mark.parametrize("nx,nr", [(3, 1), (5, 3)])
@pytest.mark.parametrize("limiter", ["positivity", "superbee"])
def test_generic_sizes_match_the_oracle(cuda, kind, p, q, nx, nr, limiter):
    cfg = pkg("config")
    cs = pkg("nozzle").build_case(element=kind, order=p, nx=nx, nr=nr, geometry_order=q, area_ratio=2.0,
                                  flow=cfg.FlowConditions(flux="hllc"),
                                  options=cfg.SolverOptions(cfl=0.3, limiter=limiter, tvb_constant=5.0))
    rng = np.random.default_rng(2)
    U = np.asarray(cs.initial_state()) * (1.0 + 0.02 * rng.standard_normal((cs.operators.n_elem, cs.operators.ref.n_basis, 1)))
    bk = pkg("backend").B200Backend(cs.operators, cs.flow, cs.options)
    assert type(bk).__name__ == "GenericB200Backend"
    R, wave = bk.residual(U)
    Ro, wo = orc.residual(U, cs.operators, cs.flow)
    assert rel(R, Ro) < 2e-12 and rel(wave, wo) < 2e-12
    assert rel(bk.rate(U)[0], orc.rate(U, cs.operators, cs.flow)[0]) < 2e-10
    step = orc.Stepper(cs.operators, cs.flow, cs.options)
    V, res_o = U, 0.0
    for _ in range(2):
        V, res_o = step.step(V)
    W, res = bk.run(U, 2, "ssprk3")
    assert rel(W, V) < 2e-10 and abs(res - res_o) <= 2e-10 * res_o
    low = np.array(U)
    low[::2, 0, 0] *= 0.05  # strong undershoots: the limiter scales
    low[::2, 0, 1:3] *= 4.0
    if limiter == "positivity":
        assert rel(bk.limit(low), orc.positivity(low, cs.operators, cs.flow)[0]) < 2e-10
