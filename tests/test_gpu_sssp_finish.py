"""SSSP's finish kernel: searches that end (and, on small graphs, begin) as
one label-correcting run give the oracle's distances and, as parents, the
smallest source of a tight edge -- on rows that span many chunks, paths of
many rounds, no light edges at all, ties, graphs that go through buckets
first, on every grid, with outputs pre-filled or not.  Edges beyond the
bucket ring are refused as in the buckets."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fans(rng):
    """Root -> 300 vertices -> 257 leaves each."""
    e = [(0, 1 + i) for i in range(300)] + [(1 + i, 301 + 257 * i + j) for i in range(300) for j in range(257)]
    return 301 + 257 * 300, np.array(e), 1.0 - rng.random(len(e), dtype=np.float32)


def _path(rng):
    """300 vertices in a row: 299 rounds, more than the trace holds."""
    e = [(i, i + 1) for i in range(299)]
    return 301, np.array(e), 1.0 - rng.random(len(e), dtype=np.float32)


def _heavy(rng):
    """No light edge at all."""
    e = rng.integers(0, 500, (4000, 2))
    return 500, e, (0.5 + 0.5 * rng.random(len(e))).astype(np.float32)


def _ties(rng):
    """Equal weights, duplicate edges, isolated vertices."""
    e = rng.integers(0, 200, (1500, 2))
    return 333, e, (rng.integers(1, 4, len(e)) * np.float32(0.25)).astype(np.float32)


def _kron(rng):
    """2^17 vertices, 2^22 edges: buckets first, then the finish."""
    u = v = np.zeros(1 << 22, np.int64)
    for _ in range(17):
        r = rng.random(1 << 22)
        u = u * 2 + (r >= 0.76)
        v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    return 1 << 17, np.stack([u, v], 1), 1.0 - rng.random(1 << 22, dtype=np.float32)


@pytest.mark.parametrize("make", [_fans, _path, _heavy, _ties, _kron])
@pytest.mark.parametrize("renumber", [False, True])
def test_finish_matches_oracle(cgt, oracle, make, renumber):
    n, e, w = make(np.random.default_rng(7))
    tg = cgt.TupleGraph(torch.tensor(e, device="cuda"), torch.tensor(w, device="cuda"), len(e))
    g = cgt.oned_graph_from_tuple_graph(tg, n, sssp_renumber=renumber)
    rs, col, ow = oracle.csr_build(e.astype(np.uint64), w, n)
    root = int(e[0, 0])
    od, _ = oracle.sssp(rs, col, ow, n, root)
    # the smallest source, in the search's numbering, of a tight edge into v
    num = g.sr.perm.cpu().numpy().astype(np.int64) if renumber else np.arange(n)
    src = np.repeat(np.arange(n), np.diff(rs.astype(np.int64)))
    tight = (od[src] >= 0) & ((od[src] + ow).astype(np.float32) == od[col])
    best = np.full(n, n, np.int64)
    np.minimum.at(best, col[tight], num[src[tight]])
    back = np.argsort(num)
    parent = np.where(best < n, back[np.minimum(best, n - 1)], -1)
    parent[root] = root
    s = cgt.SsspState(g)
    for prefill in (True, False):
        for blocks in (0, 1, 5):
            if prefill:
                cgt.oned_graph_sssp_reset(s)
            else:
                assert cgt.lib.g5_sssp_reset(n, None, None, s.work.data_ptr(), s.work.numel(), None) == 0
                s.dist.fill_(9.0)
                s.pred.fill_(9)
            cgt.oned_graph_sssp_traverse(g, s, root, blocks=blocks, small=False)
            cgt.sssp_status(s)
            key = (prefill, blocks)
            assert np.array_equal(s.dist.cpu().numpy().view(np.uint32), od.view(np.uint32)), key
            assert np.array_equal(s.pred.cpu().numpy(), parent), key
    kinds = set(cgt.sssp_trace(s)["kind"])
    assert 7 in kinds and (1 in kinds) == (n == 1 << 17)


def test_edges_beyond_the_ring_are_refused(cgt):
    e = torch.tensor([[0, 1], [1, 2], [2, 3]], device="cuda")
    w = torch.tensor([0.5, 7.0, 0.5], device="cuda")
    g = cgt.oned_graph_from_tuple_graph(cgt.TupleGraph(e, w, 3), 4)
    s = cgt.SsspState(g)
    for kw in (dict(), dict(pull=-1.0, sub_min=-1)):
        cgt.oned_graph_sssp_run(g, s, 0, small=False, **kw)
        with pytest.raises(cgt.G5Error):
            cgt.sssp_status(s)
    cgt.oned_graph_sssp_run(g, s, 0, small=False, delta=0.5)  # wide enough for the weights: answered
    cgt.sssp_status(s)
    assert s.dist.tolist() == [0.0, 0.5, 7.5, 8.0]
