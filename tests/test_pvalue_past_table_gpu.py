"""Groups past the end of a source's table, and on chromosomes that it has none of, take no part in its p-values,
also where their sums are infinite or not a number.  Needs a GPU."""
import numpy as np
import pytest

from riggle_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 20])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_groups_past_the_table(rows, bad):
    D = 20
    m = api.Moments(D, [5000, 5000, 5000])
    for d in range(D):
        mean = np.arange(1, m.slots(0) + 1) * 0.01 * (d + 1)
        mv = np.stack([mean, 3 * mean], 1)
        m.set(d, 0, mv[:40] if d % 2 else mv)
        if d % 3 == 0:
            m.set(d, 1, mv)
    li = np.arange(1, 81, dtype=np.uint64)
    cnt = np.full(80, 3, np.uint64)
    s = cnt * 0.9
    good = [(0, (li[:40], s[:40], s[:40] * 0.9, cnt[:40])), (2, (li, s, s * 0.9, cnt))]
    wild = [(0, (li, np.where(li > 40, bad, s), np.where(li > 40, bad, s * 0.9), cnt)),
            (1, (li, np.full(80, bad), np.full(80, bad), cnt)), (2, (li, np.full(80, bad), s, cnt))]
    counts = np.full((rows, D), 2, np.uint32)
    bp = (np.arange(rows * D, dtype=np.uint64).reshape(rows, D) + 1) * 700
    want = m.pvalues([good] * rows, counts, bp)
    got = m.pvalues([wild] * rows, counts, bp)
    for d in range(D):
        if d % 2 and d % 3:  # 40 entries on chromosome 0, none elsewhere
            assert np.array_equal(want[3][:, d], got[3][:, d])
            for a, b in zip(want[:3], got[:3]):  # (another order of a hundred terms of one sign)
                assert np.isfinite(a[:, d]).all()
                assert np.allclose(a[:, d], b[:, d], rtol=1e-9, atol=0)
