"""Searches that meet a column entry that is no vertex: reported as that and
nothing else, whatever the grid and whether buckets or the finish meet it,
with no vertex's distance touched on its account; the state is then reset and
searched again."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N = 4000


def _chain(cgt, bad):
    """Vertices 1 .. N-1 in a row, 0 isolated; `bad` in place of one entry."""
    rs = np.zeros(N + 1, np.int64)
    rs[2:] = 2  # vertices 2 .. N-2 have two neighbours, the ends one
    rs[2], rs[N] = 1, 1
    rs = np.cumsum(rs)
    col = np.concatenate([[v for v in (u - 1, u + 1) if 1 <= v < N] for u in range(1, N)]).astype(np.int32)
    if bad is not None:
        col[7] = bad
    e = len(col)
    return cgt.OnedGraph(N, e, torch.tensor(rs, device="cuda"), torch.tensor(col, device="cuda"),
                         torch.full((e,), 0.25, device="cuda"), torch.zeros(N, dtype=torch.int32, device="cuda"), 0.1)


@pytest.mark.parametrize("blocks", [0, 1, 5])
@pytest.mark.parametrize("buckets", [False, True])
def test_entry_that_is_no_vertex(cgt, blocks, buckets):
    good = _chain(cgt, None)
    s = cgt.SsspState(good)
    for bad in (N, -1):
        g = _chain(cgt, bad)
        cgt.oned_graph_sssp_reset(s)
        cgt.oned_graph_sssp_traverse(g, s, 1, blocks=blocks, small=False, check_opens=buckets)
        with pytest.raises(cgt.G5InvalidError, match=r"flags 0x2\)"):
            cgt.sssp_status(s)
        assert float(s.dist[0]) == -1.0 and int(s.pred[0]) == -1
    cgt.oned_graph_sssp_reset(s)
    cgt.oned_graph_sssp_traverse(good, s, 1, blocks=blocks, small=False, check_opens=buckets)
    cgt.sssp_status(s)
    assert np.array_equal(s.dist.cpu().numpy(), np.r_[-1.0, 0.25 * np.arange(N - 1)].astype(np.float32))
