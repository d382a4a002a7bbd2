"""smoke()'s oracle: the scene comes from sundog's own scene code; where that
was never built, and only then, from this library's derivation."""

import numpy as np
import pytest

import __graft_entry__ as entry
from oracle import oracle
from sundog_b200 import workloads


def test_missing_scene_code_leaves_the_oracle_in_place(lib, oracle_lib, monkeypatch):
    def missing():
        raise oracle.SceneCodeMissing("not built")
    monkeypatch.setattr(oracle, "ref_scene_lib", missing)
    text, r, by = entry.oracle_scene_text(workloads.cornell(width=8, height=8, spp=2), lib)
    assert by == "own" and (r["width"], r["height"], r["spp"]) == (8, 8, 2)
    osc = oracle.OracleScene(text)
    film, rays, _, _ = osc.render(0, 0, 8, 8, 0, 2)
    osc.close()
    assert np.isfinite(film).all() and film[..., :3].max() > 0 and rays > 8 * 8 * 2


def test_broken_scene_code_is_an_error(lib, monkeypatch):
    def broken(*a, **k):
        raise RuntimeError("oracle: reference scene text failed")
    monkeypatch.setattr(oracle, "ref_scene_lib", lambda: None)
    monkeypatch.setattr(oracle, "reference_scene_text", broken)
    with pytest.raises(RuntimeError, match="scene text failed"):
        entry.oracle_scene_text(workloads.cornell(width=8, height=8, spp=2), lib)
