"""Where a bucket goes on by sub-buckets by default: on graphs of 5 x 2^25
entries and more, or 9 x 2^16 a block of a smaller grid, not on smaller ones
whose frontier passes 2^22 entries, where they cost more than they save; with
the same distances and parents."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
SPLIT = 5  # trace kind


@pytest.mark.parametrize("scale,edgefactor,blocks,splits", [(20, 32, 0, False), (20, 32, 222, False), (20, 32, 55, True),
                                                            (22, 24, 0, True)])
def test_default_line(cgt, scale, edgefactor, blocks, splits):
    g = cgt.oned_graph_from_kronecker(cgt.make_mrg_seed(2, 3), scale, edgefactor << scale)
    assert (g.nlocaledges >= (min(5 << 25, blocks * (9 << 16)) if blocks else 5 << 25)) == splits
    root = int(torch.argmax(g.rowstarts[1:] - g.rowstarts[:-1]))
    s = cgt.SsspState(g)
    out = []
    for sub_min in (0, 1 << 22, -1):
        cgt.oned_graph_sssp_run(g, s, root, blocks=blocks, sub_min=sub_min, small=False)
        cgt.sssp_status(s)
        out.append((s.dist.clone(), s.pred.clone(), SPLIT in cgt.sssp_trace(s)["kind"]))
    assert [x[2] for x in out] == [splits, True, False]
    for dist, pred, _ in out[1:]:
        assert torch.equal(dist.view(torch.int32), out[0][0].view(torch.int32)) and torch.equal(pred, out[0][1])
