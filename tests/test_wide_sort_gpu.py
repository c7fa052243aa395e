"""Blocks that hold several rows (one block per shard), sorted block by block by (row, start): at the tile edges of the
sort, in and out of order, with blocks in any shard order, and with an interval whose row is out of range.
Needs a GPU."""
import numpy as np
import pytest

import oracle as O
import riggle_b200 as rg
from riggle_b200 import _lib

pytestmark = pytest.mark.gpu

SPAN, D = 4_000_000, 6


def _db(rng):
    out = []
    for sh in range(3):
        s = rng.integers(0, SPAN, 8000)
        ln = np.where(rng.random(8000) < 0.8, rng.integers(1, 900, 8000), rng.integers(1, 80_000, 8000))
        out.append((sh, np.stack([s, s + ln, rng.integers(0, D, 8000)], 1).astype(np.uint32)))
    return rg.bucket_layers(out)


@pytest.mark.parametrize("order", ["by row and start", "by start", "shuffled"])
@pytest.mark.parametrize("n", [1, 300, 4095, 4096, 4097, 8193, 30_001])
def test_rows_in_one_block(n, order):
    rng = np.random.default_rng(n)
    layers = _db(rng)
    rows = 37
    q = {}
    for sh, m in ((2, n), (0, max(1, n // 2)), (1, 17)):
        s = rng.integers(0, SPAN, m)
        b = np.stack([s, s + rng.integers(1, 3000, m), rng.integers(0, rows, m)], 1).astype(np.uint32)
        if order == "by row and start":
            b = b[np.lexsort((b[:, 0], b[:, 2]))]
        elif order == "by start":
            b = b[np.argsort(b[:, 0], kind="stable")]
        q[sh] = b
    oc, _, obp, _ = O.query_database(layers, q, rows, D, threads=4)
    idx = rg.Index.from_layers(layers, D, ["a", "b", "c"])
    ctx = rg.Context(idx)
    for ratio in (0, 1):
        c, bp, _ = ctx.query_counts(q, rows, pair_ratio=ratio)
        assert (c == oc).all() and (bp == obp).all()


def test_bad_row_is_refused_and_the_context_goes_on():
    rng = np.random.default_rng(3)
    layers = _db(rng)
    idx = rg.Index.from_layers(layers, D, ["a", "b", "c"])
    ctx = rg.Context(idx)
    s = np.sort(rng.integers(0, SPAN, 5000))
    q = np.stack([s, s + 700, np.arange(5000) // 1300], 1).astype(np.uint32)
    bad = q.copy()
    bad[4321, 2] = 9
    with pytest.raises(rg.RiggleError) as e:
        ctx.query_counts({0: bad}, 4)
    assert e.value.status == _lib.RGL_ERR_INVALID_ARGUMENT
    oc, _, obp, _ = O.query_database(layers, {0: q}, 4, D, threads=4)
    c, bp, _ = ctx.query_counts({0: q}, 4)
    assert (c == oc).all() and (bp == obp).all()
