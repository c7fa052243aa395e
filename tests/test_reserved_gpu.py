"""After Context.reserve the device and host queries allocate no device memory, blocks of several rows in any shard
order among them.  Needs a GPU."""
import ctypes as C

import numpy as np
import pytest

import helpers
import oracle as O
import riggle_b200 as rg
from riggle_b200 import _lib

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _allocations(f):
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    names = [e.key for e in p.key_averages()]
    if not any("k_expand_keys" in n for n in names):
        pytest.skip("the profiler does not see the library's calls here")
    return [n for n in names if n.startswith(("cudaMalloc", "cuMemAlloc", "cudaFree", "cuMemFree"))]


@pytest.mark.parametrize("rows", [1, 9])
@pytest.mark.parametrize("order", [(0, 1, 2), (2, 0, 1)])
def test_queries_after_reserve(rows, order):
    rng = np.random.default_rng(rows)
    db = [(sh, helpers.random_db(rng, 5000, 1_000_000, 6)) for sh in range(3)]
    layers = rg.bucket_layers(db)
    idx = rg.Index.from_layers(layers, 6, ["a", "b", "c"])
    q = {sh: helpers.queries_touching(rng, db[sh][1], 700 + sh, rows) for sh in order}
    want = O.query_database(layers, q, rows, 6, threads=2)
    warm = rg.Context(idx)  # loads the kernels
    warm.query_counts(q, rows)
    ctx = rg.Context(idx)
    ctx.reserve(5000, rows)
    iv = torch.from_numpy(np.concatenate(list(q.values())).view(np.int32)).to("cuda:0")
    off = np.concatenate([[0], np.cumsum([len(v) for v in q.values()])]).astype(np.uint64)
    counts = torch.zeros((rows, 6), dtype=torch.int32, device="cuda:0")
    bp = torch.zeros((rows, 6), dtype=torch.int64, device="cuda:0")
    ids = np.array(order, np.uint32)

    def device_call():
        _lib.check(rg.load().rgl_query_counts_device(ctx._h, rows, 3, C.c_void_p(ids.ctypes.data),
                                                     C.c_void_p(off.ctypes.data), C.c_void_p(iv.data_ptr()), None,
                                                     C.c_void_p(counts.data_ptr()), C.c_void_p(bp.data_ptr()), None))

    assert not _allocations(device_call)
    ctx.check()
    assert (counts.cpu().numpy().view(np.uint32) == want[0]).all()
    assert (bp.cpu().numpy().view(np.uint64) == want[2]).all()
    host = []
    assert not _allocations(lambda: host.append(ctx.query_counts(q, rows)))
    assert (host[0][0] == want[0]).all() and (host[0][1] == want[2]).all()
