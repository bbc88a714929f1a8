"""Top-down levels: each warp's first grab and chunk are its own number's and
the rest come from counters.  Lists shorter and longer than the grid's
warps, rows around the chunk size, and grids from one block to the whole
device give the oracle's depths and a valid tree."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fans(width, rows):
    """Root -> `rows` vertices -> `width` leaves each: levels of 1, rows and rows * width vertices."""
    e = [(0, 1 + i) for i in range(rows)]
    n = 1 + rows
    for i in range(rows):
        e += [(1 + i, n + j) for j in range(width)]
        n += width
    return n + 5, e  # and five isolated vertices


@pytest.mark.parametrize("width,rows", [(1, 1), (127, 3), (128, 40), (129, 40), (257, 300), (3, 5000), (20000, 2)])
def test_top_down_lists(cgt, oracle, width, rows):
    n, e = _fans(width, rows)
    e = np.array(e, np.int64)
    w = np.full(len(e), 0.5, np.float32)
    g = cgt.oned_graph_from_tuple_graph(cgt.TupleGraph(torch.tensor(e, device="cuda"), torch.tensor(w, device="cuda"),
                                                       len(e)), n, sssp_renumber=False)
    rs, col, _ = oracle.csr_build(e.astype(np.uint64), w, n)
    bfs = cgt.BfsState(g)
    _, most = cgt.search_grid("bfs", n)
    for root in (0, 1, n - 6, n - 1):
        _, depth = oracle.bfs(rs, col, n, root)
        for mode in (0, 1):
            for blocks in (0, 1, 2, 37, most):
                for tiles in ((0, 0), (32, 32), (1 << 20, 65536)):
                    cgt.oned_graph_bfs_reset(bfs, True, g)
                    cgt.oned_graph_bfs_traverse(g, bfs, root, cgt.BfsParams(14.0, 24.0, mode, blocks, *tiles))
                    st = cgt.bfs_stats(bfs)
                    key = (root, mode, blocks, tiles)
                    assert np.array_equal(bfs.depth.cpu().numpy(), depth), key
                    assert st.reached == int((depth >= 0).sum()), key
        dist = cgt.bfs_compute_dist_from_pred(g, bfs, root)
        assert cgt.bfs_validate(g, root, bfs.pred, dist) == 0
