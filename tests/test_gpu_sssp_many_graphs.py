"""Packed graphs with 2^30 entries and more in all are searched in buckets to
the end, fewer are handed to the finish; each graph's distances are those of
the graph searched alone."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
FINISH = 7  # trace kind


@pytest.mark.parametrize("scales,finish", [([12, 18, 18], True), ([20] * 33 + [12, 14], False)])
def test_finish_by_entries(cgt, scales, finish):
    pk = cgt.pack_kronecker(scales, edgefactor=16, seed1_base=100, seed2=3, device="cuda")
    assert (pk.g.nlocaledges < 1 << 30) == finish
    s = cgt.SsspState(pk.g)
    buckets = []
    for pull in (1.0, 0.0):  # the default's value asks for buckets to the end, 0 for the default
        cgt.oned_graph_sssp_reset(s)
        cgt.oned_graph_sssp_traverse_multi(pk.g, s, pk.d_roots, pull=pull)
        buckets.append(cgt.sssp_status(s)[0])
    assert (buckets[1] < buckets[0]) == finish and (buckets[1] == buckets[0]) != finish
    kinds = cgt.sssp_trace(s)["kind"]
    assert (FINISH in kinds) == finish or len(kinds) == 256
    for i in (0, len(scales) - 1):
        g = cgt.oned_graph_from_kronecker(cgt.make_mrg_seed(100 + i, 3), scales[i], 16 << scales[i], with_main=False)
        one = cgt.SsspState(g)
        cgt.oned_graph_sssp_run(g, one, int(pk.local_roots[i]), small=False)
        cgt.sssp_status(one)
        assert np.array_equal(s.dist[pk.graph_slice(i)].cpu().numpy().view(np.uint32),
                              one.dist.cpu().numpy().view(np.uint32))
