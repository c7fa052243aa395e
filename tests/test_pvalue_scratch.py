"""The scratch that the p-values of up to so many rows take: never less for more rows (the request server forms its
batches by that).  Needs no GPU."""
import pytest

import riggle_b200 as rg


@pytest.mark.parametrize("chroms", [1, 2, 24, 64, 65, 455])
def test_scratch_never_falls(chroms):
    f = rg.load().rgl_pvalue_scratch_bytes
    for sources in list(range(1, 200, 7)) + [500, 1169, 1905, 3000, 5585, 6000, 9456, 9457, 40_000]:
        sizes = [f(r, sources, chroms) for r in range(1, 1200)]
        assert all(a <= b for a, b in zip(sizes, sizes[1:])), sources
        # a launch of `r` rows is split where its tiles are fewer than 592, and then holds its cells' sums apart
        for r in (1, 4, 15, 16, 17, 128, 256, 1199):
            tiles = -(-r // (32 if r >= 16 else 4)) * -(-sources // 16)
            if tiles < 592 and 1 < chroms <= 64:
                assert sizes[r - 1] >= 25 * r * sources * chroms
    assert f(0, 100, chroms) <= 64


def test_scratch_is_bounded():
    f = rg.load().rgl_pvalue_scratch_bytes
    for chroms, most in ((24, 200 << 20), (64, 500 << 20), (1_000_000, 200 << 20)):
        assert max(f(r, s, chroms) for r in (1, 15, 128, 5000) for s in (1, 500, 20_000)) <= most
