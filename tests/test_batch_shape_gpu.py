"""The launch shape of a batch: a default and the value it stands for are two shapes, also for the kept graph.  Needs a
GPU."""
import numpy as np
import pytest

import helpers
import oracle as O
import riggle_b200 as rg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

ROWS, D, SPAN = 12, 19, 2_000_000


@pytest.fixture(scope="module")
def setup():
    rng = np.random.default_rng(8)
    db = [(sh, helpers.random_db(rng, 20_000, SPAN, D)) for sh in range(2)]
    layers = rg.bucket_layers(db)
    parts, shards, rows, per = [], [], [], {0: [], 1: []}
    for r in range(ROWS):
        for sh in range(2):
            q = helpers.random_db(rng, int(rng.integers(50, 3000)), SPAN, 1)
            q[:, 2] = r
            parts.append(q)
            shards.append(sh)
            rows.append(r)
            per[sh].append(q)
    want = O.query_database(layers, {sh: np.concatenate(v) for sh, v in per.items()}, ROWS, D, threads=4)
    iv = torch.from_numpy(np.concatenate(parts).view(np.int32)).to("cuda:0")
    off = np.concatenate([[0], np.cumsum([len(p) for p in parts])]).astype(np.uint64)
    idx = rg.Index.from_layers(layers, D, ["a", "b"])
    return idx, rg.DeviceBatch(ROWS, shards, off, iv.data_ptr(), rows), iv, want


def _run(ctx, batch, want, **kw):
    c = torch.zeros((ROWS, D), dtype=torch.int32, device="cuda:0") if "c" not in kw else kw.pop("c")
    bp = torch.zeros((ROWS, D), dtype=torch.int64, device="cuda:0") if "bp" not in kw else kw.pop("bp")
    st = ctx.query_batch_device(batch, c.data_ptr(), bp.data_ptr(), **kw)
    assert (c.cpu().numpy().view(np.uint32) == want[0]).all() and (bp.cpu().numpy().view(np.uint64) == want[2]).all()
    return st


@pytest.mark.parametrize("given", [dict(pair_ratio=4), dict(chunk=1024)])
def test_graph_of_a_default_is_not_that_of_its_value(setup, given):
    idx, batch, _, want = setup
    ctx = rg.Context(idx)
    out = dict(c=torch.zeros((ROWS, D), dtype=torch.int32, device="cuda:0"),
               bp=torch.zeros((ROWS, D), dtype=torch.int64, device="cuda:0"))
    plain = _run(ctx, batch, want, **given)
    assert _run(ctx, batch, want, graph=True, **out)["graph_replayed"] == 0
    assert _run(ctx, batch, want, graph=True, **out)["graph_replayed"] == 1
    st = _run(ctx, batch, want, graph=True, **out, **given)
    assert st["graph_replayed"] == 0
    for key in ("rank_positions", "pair_candidates", "ranges"):
        assert st[key] == plain[key]
    assert _run(ctx, batch, want, graph=True, **out, **given)["graph_replayed"] == 1


def test_tuned_shape_is_one_that_was_tried(setup):
    idx, batch, _, want = setup
    ctx = rg.Context(idx)
    by_ratio = {r: _run(ctx, batch, want, pair_ratio=0 if r == 4 else r) for r in (1, 2, 4, 8)}
    given = _run(ctx, batch, want, pair_ratio=4)
    assert given["rank_positions"] != by_ratio[4]["rank_positions"]  # the default is not the ratio alone
    best, trials = ctx.autotune(batch)
    assert len(trials) == 29
    st = _run(ctx, batch, want, tuned=True)
    assert (st["chunk"], st["ctas_per_sm"], st["pair_ratio"]) == (best["chunk"], best["ctas_per_sm"], best["pair_ratio"])
    for key in ("rank_positions", "pair_candidates"):
        assert st[key] == by_ratio[best["pair_ratio"]][key]
