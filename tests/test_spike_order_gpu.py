"""The impulses of one bin are summed in input order, starts before ends, whatever the order of the intervals and
whatever the key bits that the number of bins needs.  Needs a GPU."""
import numpy as np
import pytest

import oracle as O
from riggle_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_bins", [2, 255, 256, 257, 65_535, 65_536, 65_537, 1 << 20])
@pytest.mark.parametrize("bin_size", [1, 64, 100])
def test_many_impulses_in_few_bins_bit_exact(n_bins, bin_size):
    rng = np.random.default_rng(n_bins + bin_size)
    n, span = 5000, n_bins * bin_size
    hot = rng.integers(0, span, 7)  # most ends share a handful of bins; some lie past the last bin
    s = np.where(rng.random(n) < 0.8, hot[rng.integers(0, 7, n)], rng.integers(0, span, n)).astype(np.int64)
    e = s + rng.integers(1, 5 * bin_size + 2, n)
    g = api.depth_signal(np.stack([s, e, np.zeros(n)], 1).astype(np.uint32), n_bins, bin_size)
    want = O.depth_signal(s.astype(np.uint32), e.astype(np.uint32), n_bins, bin_size)
    assert (g == want).all()
