"""bfs_compute_dist_from_pred's edge-parallel parent check and chain walk:
the reference's distances (the oracle's restatement) on rows that span many
tiles, runs of empty rows, trees deeper than one pass walks, and parents that
are no edge, no vertex, their own child or part of a cycle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _path(n):
    return n + 3, [(i, i + 1) for i in range(n - 1)]


def _hubs(n):
    """Two joined hubs with n leaves each, every tenth vertex isolated."""
    leaf = [v for v in range(2, 5 * n) if v % 10][:2 * n]
    return 5 * n, [(0, 1)] + [(0, v) for v in leaf[:n]] + [(1, v) for v in leaf[n:]]


def _random(n):
    e = np.random.default_rng(n).integers(0, n, (4 * n, 2))
    return 4 * n, [tuple(x) for x in e if x[0] != x[1]]  # three quarters isolated


@pytest.mark.parametrize("graph", [_path(2), _path(64), _path(65), _path(300), _hubs(31), _hubs(3000), _random(1024),
                                   _random(5000)])
def test_dist_from_pred_matches_oracle(cgt, oracle, graph):
    n, e = graph
    e = np.array(e, np.int64).reshape(-1, 2)
    w = np.full(len(e), 0.5, np.float32)
    g = cgt.oned_graph_from_tuple_graph(cgt.TupleGraph(torch.tensor(e, device="cuda"), torch.tensor(w, device="cuda"),
                                                       len(e)), n, sssp_renumber=False)
    rs, col, _ = oracle.csr_build(e.astype(np.uint64), w, n)
    bfs = cgt.BfsState(g)
    root = int(e[0, 0]) if len(e) else 0
    cgt.oned_graph_bfs_run(g, bfs, root)
    good = bfs.pred.cpu().numpy().copy()
    rng = np.random.default_rng(1)
    for what in range(6):
        pred = good.copy()
        hit = rng.permutation(n)[: max(1, n // 8)]
        if what == 1:
            pred[hit] = rng.integers(0, n, len(hit))  # mostly no edge
        elif what == 2:
            pred[hit] = hit  # their own parents
        elif what == 3:
            pred[hit] = n + 7  # no vertex
        elif what == 4 and len(e):
            pred[e[:, 0]], pred[e[:, 1]] = e[:, 1], e[:, 0]  # cycles of two
        elif what == 5:
            pred[hit] = -1
        bfs.pred.copy_(torch.from_numpy(pred))
        got = cgt.bfs_compute_dist_from_pred(g, bfs, root).cpu().numpy()
        assert np.array_equal(got, oracle.bfs_dist_from_pred(rs, col, n, pred, root)), what
