"""P-values of genomes of many chromosomes, on both sides of the line (64) beyond which a warp takes a cell: the bits of
the same rows alone, and the sums of the groups.  Needs a GPU."""
import numpy as np
import pytest

from riggle_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [64, 65, 3000])
@pytest.mark.parametrize("rows,D", [(128, 30), (200, 160), (9, 31)])
def test_many_chromosomes(rows, D, C):
    bins = 300
    rng = np.random.default_rng(rows)
    m = api.Moments(D, [bins] * C)
    lens = np.arange(1, m.slots(0) + 1)
    table = {}
    for d in range(D):
        for c in rng.choice(C, min(C, 40), replace=False):
            mean = (lens * rng.uniform(0.01, 0.4)).astype(np.float32)
            var = (mean * rng.uniform(0.4, 9.0)).astype(np.float32)
            m.set(d, int(c), np.stack([mean, var], 1))
            table[d, int(c)] = (mean, var)
    rowg = []
    for q in range(rows):
        per = []
        for c in np.sort(rng.choice(C, 3 * C // 10, replace=False)):
            li = np.unique(rng.integers(1, 100, 3)).astype(np.uint64)
            cnt = rng.integers(1, 9, len(li)).astype(np.uint64)
            per.append((int(c), (li, cnt * 0.9, cnt * 0.85, cnt)))
        rowg.append(per)
    counts = rng.integers(1, 3, (rows, D)).astype(np.uint32)
    bp = rng.integers(1, 200_000, (rows, D)).astype(np.uint64)
    whole = m.pvalues(rowg, counts, bp)
    for q in (0, rows // 2, rows - 1):
        alone = m.pvalues(rowg[q:q + 1], counts[q:q + 1], bp[q:q + 1])
        for a, b in zip(alone, whole):
            assert np.array_equal(a[0], b[q])
    seen = 0
    for q, d in zip(rng.integers(0, rows, 30), rng.integers(0, D, 30)):
        mu = var = raw = 0.0
        for c, (li, ss, ss2, cnt) in rowg[q]:
            if (d, c) in table:
                mean, v = (t[li.astype(int) - 1].astype(np.float64) for t in table[d, c])
                mu, var, raw = mu + (mean * ss).sum(), var + (v * ss2).sum(), raw + (mean / li * cnt).sum()
        assert bool(whole[3][q, d] & 1) == (raw > 0)
        if raw > 0 and var > mu and whole[3][q, d] & 2:
            obs = bp[q, d] / 100.0
            r, p, po = mu * mu / (var - mu), mu / var, mu * mu / (var - mu) / (mu * mu / (var - mu) + obs)
            # each sum is within n * 2^-53 of itself (n < 3,000 terms, all positive): 3e-13; var - mu, 1 - p and
            # 1 - po cancel a few digits of that, and the two terms of the ratio may cancel each other
            a, b = obs * np.log((1 - po) / (1 - p)), r * np.log(po / p)
            assert abs(whole[1][q, d] - (a + b)) <= 1e-10 * (abs(a) + abs(b) + r + obs)
            seen += 1
    assert seen
    m.close()
