"""The request server with the statistics stage over many sources, and more requests pending than a batch takes: sizes
at which the p-values of a full batch need no scratch and those of a few requests do.  Every request is answered, and
with the bits it gets alone.  Needs a GPU."""
import threading

import numpy as np
import pytest

import riggle_b200 as rg
from riggle_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,most", [(1905, 256), (5585, 16)])
def test_a_burst_is_answered(D, most):
    rng = np.random.default_rng(D)
    n = 4000
    s = rng.integers(0, 150_000, n)
    db = np.stack([s, s + rng.integers(1, 2000, n), rng.integers(0, D, n)], 1).astype(np.uint32)
    idx = rg.Index.from_layers(rg.bucket_layers([(0, db), (1, db[::-1].copy())]), D, ["a", "b"])
    m = api.Moments(D, [2000] * 24)
    for d in range(D):
        mean = np.arange(1, m.slots(0) + 1) * float(rng.uniform(0.001, 0.3))
        m.set(d, d % 2, np.stack([mean, mean * float(rng.uniform(0.5, 9.0))], 1))
    reqs = []
    for k in range(most + 200):
        q = rng.integers(0, 150_000, int(rng.integers(5, 40)) if k else 200)
        iv = np.stack([q, q + rng.integers(1, 3000, len(q)), np.zeros_like(q)], 1).astype(np.uint32)
        reqs.append({0: iv, 1: iv[: len(iv) // 2]})
    gate = threading.Event()
    gate.set()

    def free():
        gate.wait(60)
        return 64 << 30

    # the first request is larger than what the worker reserved, so the worker asks for the free memory, and waits
    # there until the whole burst is queued
    srv = rg.Server(idx, workers=1, max_batch_requests=most, batch_intervals=50_000, initial_intervals=100,
                    free_memory=free, moments=m, shard_chrom=[0, 1])
    gate.clear()
    tickets = [srv.submit(r) for r in reqs]
    gate.set()
    mix = [srv.wait(t, timeout_ms=30_000) for t in tickets]
    assert max(info["batch_requests"] for _, _, info in mix) == most
    assert srv.stats()["failed"] == 0
    some = 0
    for k in range(0, len(reqs), 37):
        c, bp, info = srv.wait(srv.submit(reqs[k]), timeout_ms=30_000)
        assert (c == mix[k][0]).all() and (bp == mix[k][1]).all()
        for key in ("p", "llr", "lp", "flags"):
            assert np.array_equal(info["pvalues"][key], mix[k][2]["pvalues"][key])
        some += int((info["pvalues"]["flags"] & 2).sum())
    assert some
    srv.close()
    m.close()
    idx.close()
