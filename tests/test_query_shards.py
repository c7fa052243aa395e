"""The shards of a host query as the library receives them.  Needs no GPU."""
import numpy as np
import pytest

from riggle_b200 import Context


@pytest.mark.parametrize("key", [0, 23, -1, 2**32 - 1, 2**32 + 5, -(2**40) - 7, np.int64(-2), np.uint64(2**63), 3.0])
def test_any_number_is_taken_as_32_bits(key):
    iv = np.array([[5, 9, 0], [7, 8, 1]], np.uint32)
    keep = []
    b = Context._batch({key: iv, "chr1": iv[:1], "none": iv[:0]}, 2, keep)
    assert b.num_rows == 2 and b.num_shards == 3
    assert b.shards[0].shard_id == int(key) % 2**32 and b.shards[0].shard_name is None and b.shards[0].count == 2
    assert b.shards[1].shard_name == b"chr1" and b.shards[1].count == 1
    assert b.shards[2].count == 0
