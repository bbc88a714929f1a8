"""Where a bucket goes on by sub-buckets by default: on graphs of 5 x 2^25
entries and more, not on smaller ones whose frontier passes 2^22 entries,
where they cost more than they save; with the same distances and parents."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
SPLIT = 5  # trace kind


@pytest.mark.parametrize("scale,edgefactor,splits", [(20, 32, False), (22, 24, True)])
def test_default_line(cgt, scale, edgefactor, splits):
    g = cgt.oned_graph_from_kronecker(cgt.make_mrg_seed(2, 3), scale, edgefactor << scale)
    assert (g.nlocaledges >= 5 << 25) == splits
    root = int(torch.argmax(g.rowstarts[1:] - g.rowstarts[:-1]))
    s = cgt.SsspState(g)
    out = []
    for sub_min in (0, 1 << 22, -1):
        cgt.oned_graph_sssp_run(g, s, root, sub_min=sub_min, small=False)
        cgt.sssp_status(s)
        out.append((s.dist.clone(), s.pred.clone(), SPLIT in cgt.sssp_trace(s)["kind"]))
    assert [x[2] for x in out] == [splits, True, False]
    for dist, pred, _ in out[1:]:
        assert torch.equal(dist.view(torch.int32), out[0][0].view(torch.int32)) and torch.equal(pred, out[0][1])
