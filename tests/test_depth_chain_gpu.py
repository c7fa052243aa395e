"""The depth signal's carry chain at the edges of its stages (2,048 totals) and steps (16), with and without tail bins
past the last chunk of eight, dense and sparse.  Needs a GPU."""
import numpy as np
import pytest

import oracle as O
from riggle_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", [0, 1, 7])
@pytest.mark.parametrize("chunks", [1, 2, 15, 17, 2047, 2048, 2049, 4097, 20_000])
def test_chain_bit_exact(chunks, tail):
    n_bins = 8 * chunks + tail
    rng = np.random.default_rng(n_bins)
    for n in (max(1, chunks // 50), 12 * chunks):  # a few chunks with a total, then almost all of them
        s = rng.integers(0, n_bins * 100, n).astype(np.int64)
        e = s + rng.integers(1, 3000, n)
        g = api.depth_signal(np.stack([s, e, np.zeros(n)], 1).astype(np.uint32), n_bins)
        want = O.depth_signal(s.astype(np.uint32), e.astype(np.uint32), n_bins)
        assert (g == want).all()
