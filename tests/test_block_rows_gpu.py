"""A batch whose blocks carry rows, with intervals that carry another one: refused, also where every second interval
of a block sorted by start is wrong, and the context then answers the corrected batch as the oracle does.  Needs a GPU."""
import numpy as np
import pytest

import oracle as O
import riggle_b200 as rg
from riggle_b200 import _lib

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SPAN, D, SHARDS = 3_000_000, 9, 2


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("per_block", [31, 4096, 5000])
@pytest.mark.parametrize("wrong", ["every second", "the last", "past the rows"])
def test_wrong_rows_are_refused(per_block, wrong, graph):
    rng = np.random.default_rng(per_block)
    db = []
    for sh in range(SHARDS):
        s = rng.integers(0, SPAN, 20_000)
        ln = np.where(rng.random(20_000) < 0.7, rng.integers(1, 900, 20_000), rng.integers(1, 90_000, 20_000))
        db.append((sh, np.stack([s, s + ln, rng.integers(0, D, 20_000)], 1).astype(np.uint32)))
    layers = rg.bucket_layers(db)
    rows = 5
    parts, shards, blk_rows, per_shard = [], [], [], {sh: [] for sh in range(SHARDS)}
    for r in range(rows):
        for sh in range(SHARDS):
            s = np.sort(rng.integers(0, SPAN, per_block))
            iv = np.stack([s, s + rng.integers(1, 4000, per_block), np.full(per_block, r)], 1).astype(np.uint32)
            parts.append(iv)
            shards.append(sh)
            blk_rows.append(r)
            per_shard[sh].append(iv)
    good = np.concatenate(parts)
    off = np.arange(len(parts) + 1, dtype=np.uint64) * per_block
    bad = good.copy()
    if wrong == "every second":
        bad[1::2, 2] = (bad[1::2, 2] + 1) % rows
    elif wrong == "the last":
        bad[per_block - 1::per_block, 2] = rows - 1 - bad[per_block - 1::per_block, 2]
    else:
        bad[::3, 2] = rows + 7
    idx = rg.Index.from_layers(layers, D, ["a", "b"])
    ctx = rg.Context(idx)
    c = torch.zeros((rows, D), dtype=torch.int32, device="cuda:0")
    bp = torch.zeros((rows, D), dtype=torch.int64, device="cuda:0")
    keep = [torch.from_numpy(a.view(np.int32)).to("cuda:0") for a in (bad, good)]
    for t, ok in ((keep[0], False), (keep[1], True), (keep[0], False), (keep[1], True)):
        b = rg.DeviceBatch(rows, shards, off, t.data_ptr(), blk_rows)
        if not ok:
            with pytest.raises(rg.RiggleError) as e:
                ctx.query_batch_device(b, c.data_ptr(), bp.data_ptr(), graph=graph)
            assert e.value.status == _lib.RGL_ERR_INVALID_ARGUMENT
            continue
        ctx.query_batch_device(b, c.data_ptr(), bp.data_ptr(), graph=graph)
        want = O.query_database(layers, {sh: np.concatenate(v) for sh, v in per_shard.items()}, rows, D, threads=4)
        assert (c.cpu().numpy().view(np.uint32) == want[0]).all()
        assert (bp.cpu().numpy().view(np.uint64) == want[2]).all()
