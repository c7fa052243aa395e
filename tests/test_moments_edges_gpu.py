"""Window moments at the edges of the tiles that the prefix sums are taken over (1,024 and 2,048 elements), of the
transforms' radices and of the directly reduced windows (65,536), in both precisions.  Needs a GPU."""
import numpy as np
import pytest

import oracle as O
from riggle_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("n_bins", [2, 3, 5, 9, 16, 17, 33, 100, 255, 257, 511, 513, 1023, 1024, 1025, 2047, 2048, 2049,
                                    4097, 16_385, 65_535, 65_537, 70_000, 131_073])
def test_moments_at_tile_edges(n_bins, precision):
    rng = np.random.default_rng(n_bins)
    n = max(2, n_bins // 10)
    s = np.sort(rng.integers(0, n_bins * 100, n)).astype(np.int64)
    e = s + rng.integers(1, 2500, n)
    iv = np.stack([s, e, np.zeros(n)], 1).astype(np.uint32)
    m = api.Moments(1, [n_bins])
    mean, var = m.build(0, 0, iv, report=True, precision=precision)
    g = O.depth_signal(iv[:, 0], iv[:, 1], n_bins)
    grid = O.moment_grid(n_bins)
    assert len(mean) == len(grid)
    sel = np.unique(np.concatenate([np.arange(min(4, len(grid))), np.arange(0, len(grid), 29), [len(grid) - 1]]))
    em, ev = O.moments_exact(g, grid[sel], threads=0)
    # the bounds that tests/test_moments_gpu.py holds both precisions to
    scale = np.maximum(np.abs(ev), 1e-12 * em * em + 1e-300)
    assert (np.abs(var[sel] - ev) / scale).max() < 1e-6
    assert (np.abs(mean[sel] - em) / np.maximum(np.abs(em), 1e-300)).max() < (1e-9 if precision == "fp64" else 1e-6)
