"""Batched SSSP takes a row's entries in batches: rows of every length around
a batch and a warp step, each with every source count's remainder, give the
oracle's distances."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 7, 32])
def test_rows_of_every_length(cgt, oracle, k):
    rng = np.random.default_rng(k)
    e = []  # a chain of hubs, hub i with i leaves
    hubs = 70
    n = hubs
    for i in range(hubs):
        if i:
            e.append((i - 1, i))
        for _ in range(i):
            e.append((i, n))
            n += 1
    e = np.array(e, np.int64)
    w = rng.random(len(e), dtype=np.float32)
    g = cgt.oned_graph_from_tuple_graph(cgt.TupleGraph(torch.tensor(e, device="cuda"), torch.tensor(w, device="cuda"),
                                                       len(e)), n)
    rs, col, ow = oracle.csr_build(e.astype(np.uint64), w, n)
    src = [int(x) for x in rng.choice(n, k, replace=False)]
    dist, _, _ = cgt.oned_graph_sssp_multi(g, src)
    for s, r in enumerate(src):
        od, _ = oracle.sssp(rs, col, ow, n, r)
        assert np.array_equal(dist[s].cpu().numpy().view(np.uint32), od.view(np.uint32)), s
