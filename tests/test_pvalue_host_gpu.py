"""The host form of the p-values: groups in any order, and calls of several threads on one store.  Needs a GPU."""
import threading

import numpy as np
import pytest

import test_pvalues_gpu as base

pytestmark = pytest.mark.gpu


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("rows,D", [(1, 7), (9, 40), (40, 70)])
def test_groups_in_any_order(rows, D):
    rng = np.random.default_rng(rows)
    m, _, groups, _, counts, bp = base.random_case(rng, rows, D)
    want = m.pvalues(groups, counts, bp)
    # chromosomes backwards (each one's lengths ascending), and the lengths of a chromosome backwards too
    assert _same(m.pvalues([row[::-1] for row in groups], counts, bp), want)
    mixed = m.pvalues([[(c, tuple(x[::-1] for x in g)) for c, g in row[::-1]] for row in groups], counts, bp)
    assert np.array_equal(mixed[3], want[3])
    # (lengths that share a table entry add up in the order they come in: 1,000 terms of one sign, a rounding each,
    # before the terms of the ratio cancel)
    assert np.allclose(mixed[1], want[1], rtol=1e-9, atol=1e-9)


def test_several_threads_on_one_store():
    rng = np.random.default_rng(5)
    m, _, groups, _, counts, bp = base.random_case(rng, 60, 90)
    want = m.pvalues(groups, counts, bp)
    errors = []

    def run(k):
        r = np.random.default_rng(k)
        for _ in range(12):
            a, b = sorted(r.integers(0, 61, 2))
            if a == b:
                continue
            got = m.pvalues(groups[a:b], counts[a:b], bp[a:b])
            if not _same(got, [w[a:b] for w in want]):
                errors.append((k, a, b))

    ts = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
