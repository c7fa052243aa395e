"""P-values of batches whose rows and sources alone fill the chip, so that a block walks all chromosomes: the bits of
the same rows taken few at a time (a block per chromosome), and the oracle's values.  Needs a GPU."""
import numpy as np
import pytest

import test_pvalues_gpu as base

pytestmark = pytest.mark.gpu


# 592 tiles (rows by 32, or by 4 below 16 rows, times sources by 16) and just above and below
@pytest.mark.parametrize("rows,D", [(512, 592), (480, 592), (33, 4737), (15, 2353), (16, 9473)])
def test_one_block_for_all_chromosomes(rows, D):
    rng = np.random.default_rng(rows + D)
    m, tables, groups, oracle_groups, counts, bp = base.random_case(rng, rows, D)
    whole = m.pvalues(groups, counts, bp)
    for q in (0, rows // 2, rows - 1):
        alone = m.pvalues(groups[q:q + 1], counts[q:q + 1], bp[q:q + 1])
        for a, b in zip(alone, whole):
            assert np.array_equal(a[0], b[q])
    checked = 0
    for q, d in zip(rng.integers(0, rows, 40), rng.integers(0, D, 40)):
        want = base.oracle_cell(oracle_groups[q], tables, d, float(bp[q, d]) / 100.0) if counts[q, d] else None
        if want is None:
            assert whole[3][q, d] == 0 and whole[0][q, d] == 1.0
            continue
        checked += 1
        if want[1] is not None:
            assert whole[1][q, d] == pytest.approx(want[1], rel=1e-9, abs=1e-12)
        if want[0] > 1e-290:
            assert whole[0][q, d] == pytest.approx(want[0], rel=1e-9)
    assert checked > 10
