"""The tuner's tiles on the CPU, with made-up times: the library's defaults are
among the candidates and win when they are the fastest, and every default of
the library can be chosen by its value."""
from __future__ import annotations

import types

import pytest


@pytest.fixture
def tuner(cgt, monkeypatch):
    from cgt_b200 import autotune as T
    cost = {}
    for name in ("BfsState", "SsspState"):
        monkeypatch.setattr(T, name, lambda g: None)
    monkeypatch.setattr(T, "_timed", lambda run, reset=None: run())
    monkeypatch.setattr(T, "oned_graph_bfs_traverse", lambda g, st, r, p, **kw: cost["of"](
        {"chunk": p.chunk, "big_deg": p.big_deg, "lane_entries": p.lane_entries}))
    monkeypatch.setattr(T, "oned_graph_sssp_traverse", lambda g, st, r, delta, blocks, pull, sub, **kw: cost["of"](kw))
    return T, cost, types.SimpleNamespace(nglobalverts=1000)


def _tune(T, kind, g):
    if kind == "bfs":
        return T.tune_bfs(g, [0], alphas=(14.0,), betas=(24.0,), grids=(0,)), T.BFS_TILES
    return T.tune_sssp(g, [0], deltas=(0.1,), grids=(0,)), T.SSSP_TILES


@pytest.mark.parametrize("kind", ["bfs", "sssp"])
def test_defaults_win_when_fastest(tuner, kind):
    T, cost, g = tuner
    cost["of"] = lambda tiles: 1.0 if not any(tiles.values()) else 2.0
    best, axes = _tune(T, kind, g)
    assert {k: best[k] for k in axes} == dict.fromkeys(axes, 0) and best["ms"] == 1.0


@pytest.mark.parametrize("kind,want", [("bfs", {"chunk": 128, "big_deg": 256, "lane_entries": 16}),
                                       ("sssp", {"chunk": 64, "big_deg": 64}), ("sssp", {"chunk": 256, "big_deg": 128})])
def test_defaults_can_be_chosen_by_value(tuner, kind, want):
    T, cost, g = tuner
    cost["of"] = lambda tiles: 10.0 - sum(tiles[k] == v for k, v in want.items())
    best, axes = _tune(T, kind, g)
    assert {k: best[k] for k in axes} == want
