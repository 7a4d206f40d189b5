"""The batch's tail: the march object is rebuilt for the single-solve kernels only where these are other ones."""

from __future__ import annotations

import json

import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


def _run(monkeypatch, path):
    cfg, batch = pkg("config"), pkg("batch")
    if path:
        monkeypatch.setenv("NZB_VARIANTS_FILE", path)
    insts = []
    for kind, tol in (("tri", 1e30), ("quad", 1e-30), ("tri", 1e-30)):
        opts = cfg.SolverOptions(cfl=0.2, tolerance=tol, max_iterations=7, check_interval=2, print_interval=0)
        cs = pkg("nozzle").build_case(element=kind, order=1, refine=0, area_ratio=2.0,
                                      flow=cfg.FlowConditions(flux="hllc"), options=opts)
        insts.append(batch.Instance(cs.operators, cs.flow, opts, cs.initial_state(), cs.geometry.length, cs.geometry))
    solver = batch.BatchSolver(insts, compact=False)
    solver.run()
    assert [r.iterations for r in solver.results()] == [1, 7, 7]
    return solver


def test_no_switch_between_equal_kernels(cuda, monkeypatch, tmp_path):
    every = {f"{k}:{o}": "split4" if o else "t1" for k in ("tri", "quad") for o in range(4)}
    path = tmp_path / "same.json"
    path.write_text(json.dumps({"choice": every, "batch_choice": every}))
    solver = _run(monkeypatch, str(path))
    assert solver.tail_switched_at is None and solver.compactions == 0


def test_switch_to_other_kernels(cuda, monkeypatch, tmp_path):
    every = {f"{k}:{o}": "split4" if o else "t1" for k in ("tri", "quad") for o in range(4)}
    single = dict(every, **{"quad:1": "t1"})
    path = tmp_path / "other.json"
    path.write_text(json.dumps({"choice": single, "batch_choice": every}))
    solver = _run(monkeypatch, str(path))
    assert solver.tail_switched_at == 1 and solver.compactions == 1
