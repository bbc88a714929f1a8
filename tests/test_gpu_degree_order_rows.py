"""g5_csr_degree_order and the vertex order: rows on both sides of every class
edge (a warp in registers, a warp in shared memory, a block, tiles and merge
passes), vertex counts around a digit and a tile, against numpy."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 31, 32, 33, 64, 65, 255, 256, 257, 511, 513, 4095, 4096, 4097, 8192, 8193, 20001, 70000]


@pytest.mark.parametrize("n", [20, 255, 256, 257, 4097, 70001])
def test_rows_of_every_class(cgt, n):
    rng = np.random.default_rng(n)
    rows = rng.permutation(n)[: len(LENGTHS)]
    length = np.zeros(n, np.int64)
    length[rows] = LENGTHS[: len(rows)]
    rs = np.concatenate([[0], np.cumsum(length)])
    e = int(rs[-1])
    col = rng.integers(0, n, e).astype(np.int32)  # any CSR: neither symmetric nor free of duplicates
    d_rs, d_col = torch.tensor(rs, device="cuda"), torch.tensor(col, device="cuda")
    g = cgt.OnedGraph(n, e, d_rs, d_col, torch.zeros(e, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda"),
                      0.1)
    cgt.oned_graph_bfs_order(g)
    place = np.empty(n, np.int64)
    place[np.argsort(-length, kind="stable")] = np.arange(n)
    src = np.repeat(np.arange(n), length)
    want = col[np.lexsort((place[col], src))]
    assert np.array_equal(g.bcol.cpu().numpy(), want)
    # the renumbered copy uses the same order; its rows are the rows, renamed
    w = rng.random(e, dtype=np.float32)
    light, tiny = rng.integers(0, 9, n).astype(np.int32), rng.integers(0, 9, n).astype(np.int32)
    g.w, g.light_deg, g.tiny_deg = (torch.tensor(x, device="cuda") for x in (w, light, tiny))
    cgt.oned_graph_sssp_renumber(g)
    inv = g.sr.inv.cpu().numpy()
    assert np.array_equal(g.sr.perm.cpu().numpy(), place) and np.array_equal(place[inv], np.arange(n))
    at = np.argsort(place[src], kind="stable")
    assert np.array_equal(g.sr.rowstarts.cpu().numpy(), np.concatenate([[0], np.cumsum(length[inv])]))
    assert np.array_equal(g.sr.col.cpu().numpy(), place[col[at]]) and np.array_equal(g.sr.w.cpu().numpy(), w[at])
    assert np.array_equal(g.sr.light_deg.cpu().numpy(), light[inv])
    assert np.array_equal(g.sr.tiny_deg.cpu().numpy(), tiny[inv])


def test_bad_column_is_reported(cgt):
    d_rs = torch.tensor([0, 2, 4], device="cuda")
    for bad in (2, -1, 2**31 - 1):
        d_col = torch.tensor([0, 1, bad, 0], dtype=torch.int32, device="cuda")
        g = cgt.OnedGraph(2, 4, d_rs, d_col, torch.zeros(4, device="cuda"),
                          torch.zeros(2, dtype=torch.int32, device="cuda"), 0.1)
        with pytest.raises(cgt.G5InvalidError):
            cgt.oned_graph_bfs_order(g)
