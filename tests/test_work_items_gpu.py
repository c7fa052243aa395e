"""Work items sized by the work: totals at the edges of a step (128 positions) and of the spread over the grid,
in one-row and several-row runs, by pairs and by ranks.  Needs a GPU."""
import numpy as np
import pytest

import oracle as O
import riggle_b200 as rg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 3])
@pytest.mark.parametrize("n", [1, 63, 127, 128, 129, 4096, 37_887, 37_889, 300_001])
def test_totals_at_item_edges(n, rows):
    # n database intervals of 100 bp side by side, and per row two queries over all of them: 2 n candidates a row
    # when swept by pairs, n positions a row when swept by rank differences
    start = (np.arange(n, dtype=np.int64) * 110 + 50).astype(np.uint32)
    db = np.stack([start, start + 100, np.arange(n) % 5], 1).astype(np.uint32)
    layers = rg.bucket_layers([(0, db)])
    end = int(start[-1]) + 300
    q = np.array([[s, e, r] for r in range(rows) for s, e in ((0, end), (70, end - 230))], np.uint32)
    oc, _, obp, _ = O.query_database(layers, {0: q}, rows, 5)
    idx = rg.Index.from_layers(layers, 5, ["a"])
    ctx = rg.Context(idx)
    for ratio in (1, 1_000_000):
        c, bp, st = ctx.query_counts({0: q}, rows, pair_ratio=ratio)
        assert (c == oc).all() and (bp == obp).all()
        assert st["rank_positions"] + st["pair_candidates"] >= n * rows
        assert st["work_items"] >= 1
