"""Result sets at the edges of the block sort's tiles of 16,384 ids: one full
tile, a remainder of one id, two full tiles, into page-locked and pageable
output and alone.  With one facility every user is in its result set."""
import numpy as np
import pytest

import rknn


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16_383, 16_384, 16_385, 32_767, 32_768, 32_769])
def test_ids_at_the_edges_of_tiles(n):
    rng = np.random.default_rng(n)
    ids = (rng.choice(2**32, size=n, replace=False).astype(np.int64) - 2**31).astype(np.int32)
    want = np.sort(ids)
    with rknn.Index(np.float32([[500, 500]]), rng.uniform(0, 1000, (n, 2)).astype(np.float32), uid=ids) as idx:
        for mode in ("fp32", "fp64"):
            for _ in range(3):
                got, off = idx.query_batch_flat(np.zeros(3, np.int32), 2, mode)
                assert np.array_equal(off, n * np.arange(4)) and np.array_equal(got, np.tile(want, 3))
            for got in idx.query_batch(np.zeros(3, np.int32), 2, mode):
                assert np.array_equal(got, want)
            assert np.array_equal(idx.query(0, 2, mode), want)
