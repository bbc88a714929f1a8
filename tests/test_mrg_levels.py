"""The generator's levels over every width: log_n on both sides of 32 (where
the endpoints change from 32 to 64 bits), edge ranges that are no multiple
of the grid, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("log_n", [1, 2, 4, 5, 6, 31, 32, 33, 40, 62])
def test_generator_levels_match_oracle(cgt, oracle, log_n):
    seed = cgt.make_mrg_seed(7 + log_n, 9)
    for start, end in ((0, 1), (5, 2501)):
        tg = cgt.generate_kronecker_range(seed, log_n, start, end)
        oe, ow = oracle.generate_kronecker_range(np.array(seed, np.uint32), log_n, start, end)
        assert np.array_equal(tg.edges.cpu().numpy().view(np.uint64), oe), (start, end)
        assert np.array_equal(tg.weights.cpu().numpy().view(np.uint32), ow.view(np.uint32)), (start, end)
