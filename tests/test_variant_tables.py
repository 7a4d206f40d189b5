"""The variant tables' precedence: a caller's table decides wherever it says something."""

from __future__ import annotations

import json
from types import SimpleNamespace

from conftest import pkg

ALL = [(k, o) for k in ("tri", "quad") for o in range(4)]


def _file(tmp_path, name, **entries):
    path = tmp_path / name
    path.write_text(json.dumps({key: {f"{k}:{o}": v for k, o in ALL} for key, v in entries.items()}))
    return str(path)


def test_a_table_of_the_callers_own_decides_for_arbitrary_states(tmp_path, monkeypatch):
    at = pkg("autotune")
    assert at.variant_for("tri", 3, "lone") == "t1"
    for name, entries, want in (("a", {"batch_choice": "split4"}, "split4"), ("b", {"choice": "t1_edge"}, "t1_edge"),
                                ("c", {"batch_choice": "split4", "lone_choice": "t1_edge"}, "t1_edge")):
        monkeypatch.setenv("NZB_VARIANTS_FILE", _file(tmp_path, name, **entries))
        assert at.variant_for("tri", 3, "lone") == want


def test_which_instances_are_arbitrary_states():
    at = pkg("autotune")
    inst = lambda n, geometry: SimpleNamespace(ops=SimpleNamespace(n_elem=n), geometry=geometry)  # noqa: E731
    assert at.arbitrary_state(inst(at.LONE_ELEMENTS + 1, None))
    assert not at.arbitrary_state(inst(at.LONE_ELEMENTS, None))
    assert not at.arbitrary_state(inst(10**6, object()))
