"""Means of the shortest lengths, in both precisions: what is left of sums of prefix sums about N / L times their
size.  Needs a GPU."""
import numpy as np
import pytest

import oracle as O
from riggle_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("n_bins", [65_537, 1 << 19, 1 << 21, (1 << 21) + 1])
def test_means_of_short_windows(n_bins, precision):
    rng = np.random.default_rng(n_bins)
    s = np.sort(rng.integers(0, n_bins * 64, 2000)).astype(np.int64)
    iv = np.stack([s, s + rng.integers(1, 2000, 2000), np.zeros(2000)], 1).astype(np.uint32)
    mean, _ = api.Moments(1, [n_bins]).build(0, 0, iv, bin_size=64, report=True, precision=precision)
    grid = O.moment_grid(n_bins)
    sel = np.arange(12)
    em, _ = O.moments_exact(O.depth_signal(iv[:, 0], iv[:, 1], n_bins, 64), grid[sel], threads=0)
    # the prefix sums are held to 2^-48 (fp32c) of the whole sum, in some 2^5 roundings, and a mean of length L
    # takes L of N of them: 2^-43 of the whole sum over N windows, against a mean of L N-ths of it; the sums over
    # them are in double-double
    assert (np.abs(mean[sel] - em) / np.abs(em)).max() < 2.0**-43 * 8
