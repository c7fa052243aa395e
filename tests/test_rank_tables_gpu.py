"""Rank tables of query segments with long empty stretches, shared bins and few queries: every range swept by rank
differences against the oracle.  Needs a GPU."""
import numpy as np
import pytest

import oracle as O
import riggle_b200 as rg

pytestmark = pytest.mark.gpu

SPAN = 40_000_000


def _queries(kind, rng):
    if kind == "one":
        s = np.array([17_000_000])
    elif kind == "same start":
        s = np.full(500, 5_000_000)
    elif kind == "two far clusters":  # one gap of most of the table between them
        s = np.concatenate([rng.integers(0, 2000, 700), rng.integers(SPAN - 4000, SPAN - 2000, 700)])
    elif kind == "steps of one bin":
        s = np.arange(3000) * 64
    else:
        s = rng.integers(0, SPAN - 100_000, 4000)
    e = s + rng.integers(1, 90_000, len(s))
    return s, e


@pytest.mark.parametrize("kind", ["one", "same start", "two far clusters", "steps of one bin", "spread"])
@pytest.mark.parametrize("rows", [1, 7])
def test_rank_sweep_with_gaps(kind, rows):
    rng = np.random.default_rng(len(kind))
    s, e = _queries(kind, rng)
    n = 60_000
    ds = rng.integers(0, SPAN, n)
    ln = np.where(rng.random(n) < 0.5, rng.integers(1, 400, n), rng.integers(1, 120_000, n))
    layers = rg.bucket_layers([(0, np.stack([ds, ds + ln, rng.integers(0, 9, n)], 1).astype(np.uint32))])
    q = np.stack([s, e, rng.integers(0, rows, len(s))], 1).astype(np.uint32)
    q = np.concatenate([q, q])  # every candidate at least twice: more candidates than the union
    oc, _, obp, ost = O.query_database(layers, {0: q}, rows, 9)
    idx = rg.Index.from_layers(layers, 9, ["a"])
    c, bp, st = rg.Context(idx).query_counts({0: q}, rows, pair_ratio=1)
    assert (c == oc).all() and (bp == obp).all()
    assert st["rank_positions"] > 0
