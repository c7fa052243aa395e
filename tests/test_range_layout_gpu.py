"""The layout of candidate runs and ranges at the edges of its tiles (256 and 1,024 queries), beyond the sizes where
tile prefixes are scanned by groups, with nested queries (a range ends with an earlier query) and with runs so long
that 32 of them pass 2^32 candidates.  Needs a GPU."""
import numpy as np
import pytest

import oracle as O
import riggle_b200 as rg

pytestmark = pytest.mark.gpu


def _check(db, q, rows, D, shards=1, ratios=(0, 1, 1_000_000)):
    layers = rg.bucket_layers([(s, db) for s in range(shards)])
    qs = {s: q for s in range(shards)}
    oc, _, obp, _ = O.query_database(layers, qs, rows, D, threads=8)
    idx = rg.Index.from_layers(layers, D, [f"s{s}" for s in range(shards)])
    ctx = rg.Context(idx)
    swept = set()
    for ratio in ratios:
        c, bp, st = ctx.query_counts(qs, rows, pair_ratio=ratio)
        assert (c == oc).all() and (bp == obp).all()
        swept.add(st["db_swept"])
    assert len(swept) == 1  # the union of the candidate runs does not depend on how it is swept
    if rows == 1:
        assert swept == {O.query_database(layers, qs, rows, D)[3]["db_swept"]}


@pytest.mark.parametrize("rows", [1, 5])
@pytest.mark.parametrize("n", [1, 31, 33, 255, 256, 257, 1023, 1024, 1025, 4099])
def test_tile_edges(n, rows):
    rng = np.random.default_rng(n)
    span = 3_000_000
    ds = rng.integers(0, span, 9000)
    db = np.stack([ds, ds + np.where(rng.random(9000) < 0.9, rng.integers(1, 700, 9000), rng.integers(1, 60_000, 9000)),
                   rng.integers(0, 7, 9000)], 1).astype(np.uint32)
    s = rng.integers(0, span, n)
    ln = np.where(rng.random(n) < 0.1, rng.integers(1, 200_000, n), rng.integers(1, 900, n))  # some hold many others
    q = np.stack([s, s + ln, rng.integers(0, rows, n)], 1).astype(np.uint32)
    _check(db, q, rows, 7, shards=3 if n < 2000 else 1)


@pytest.mark.parametrize("rows", [1, 3])
def test_grouped_prefixes(rows):
    # 2.2e6 queries: more than 2,048 tiles of 1,024 queries and of 256 entries a slot
    rng = np.random.default_rng(rows)
    span, n = 200_000_000, 2_200_000
    ds = rng.integers(0, span, 20_000)
    db = np.stack([ds, ds + rng.integers(1, 5000, 20_000), rng.integers(0, 4, 20_000)], 1).astype(np.uint32)
    s = np.sort(rng.integers(0, span, n))
    q = np.stack([s, s + rng.integers(1, 800, n), rng.integers(0, rows, n)], 1).astype(np.uint32)
    _check(db, q, rows, 4, ratios=(0, 1_000_000))


def test_runs_of_more_than_2_to_27_candidates():
    length = np.array([200_000_000], np.uint32)
    sizes = [180_000_000, 150_000_000, 1000]
    idx = rg.Index.synth(rg.SynthSpec(5, length, sizes))
    ctx = rg.Context(idx)
    q = np.array([[0, 200_000_000, 0], [1, 200_000_000, 0], [150, 199_999_000, 0], [3, 7, 0]] * 12, np.uint32)
    whole = q[[0, 1, 2] * 12]  # 36 runs over the whole of every layer
    c, _, st = ctx.query_counts({0: whole[:1]}, 1, pair_ratio=1_000_000)
    assert c[0].tolist() == sizes and st["pair_candidates"] == sum(sizes)
    by_rank, bp, _ = ctx.query_counts({0: q}, 1, pair_ratio=1)
    by_pair, bp2, st = ctx.query_counts({0: q}, 1, pair_ratio=1_000_000)
    assert (by_rank == by_pair).all() and (bp == bp2).all()
    assert st["pair_candidates"] > 30 * sum(sizes[:2]) // 2


@pytest.mark.parametrize("order", ["by start", "shuffled"])
def test_ends_sorted_only_where_a_rank_sweep_needs_them(order):
    # a run beyond 2^21 queries: shard 0 has ranges that are swept by ranks, shard 1 has none, shard 2 few queries
    rng = np.random.default_rng(8)
    m = 30_000
    wide = rng.integers(0, 2_000_000, m)
    narrow = rng.integers(0, 200_000_000, m)
    db = [(0, np.stack([wide, wide + rng.integers(40_000, 100_000, m), rng.integers(0, 5, m)], 1).astype(np.uint32)),
          (1, np.stack([narrow, narrow + rng.integers(1, 500, m), rng.integers(0, 5, m)], 1).astype(np.uint32)),
          (2, np.stack([wide, wide + rng.integers(1, 100_000, m), rng.integers(0, 5, m)], 1).astype(np.uint32))]
    layers = rg.bucket_layers(db)
    q = {}
    for sh, n, span in ((0, 3_000, 2_000_000), (1, 2_150_000, 200_000_000), (2, 40, 2_000_000)):
        s = rng.integers(0, span, n)
        s = np.sort(s) if order == "by start" else s
        q[sh] = np.stack([s, s + rng.integers(1, 900, n), np.zeros(n)], 1).astype(np.uint32)
    oc, _, obp, _ = O.query_database(layers, q, 1, 5, threads=8)
    idx = rg.Index.from_layers(layers, 5, ["a", "b", "c"])
    ctx = rg.Context(idx)
    for ratio in (0, 1, 1_000_000):
        c, bp, st = ctx.query_counts(q, 1, pair_ratio=ratio)
        assert (c == oc).all() and (bp == obp).all()
        assert (st["rank_positions"] > 0) == (ratio < 2)
