"""Result sets of every size class, sorted into each kind of output.

With one facility every user is in its result set, so a set has exactly as
many ids as there are users, whatever k: the sizes here sit at the edges of
the sort's classes (32, 64, 128, 256 and 512 ids, and the block's radix sort
beyond, by tiles of 16,384).  Beside a few hundred facilities far from every
user the same sets are few in their batch, and warps sort the large ones.
"""
import numpy as np
import pytest

import rknn

SIZES = [1, 31, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 2048, 8192, 8193, 16_385, 70_001]


def _index(n, ids, far):
    rng = np.random.default_rng(n)
    fxy = np.concatenate([[[500.0, 500.0]], rng.uniform(90_000, 100_000, (far, 2))]).astype(np.float32)
    return rknn.Index(fxy, rng.uniform(0, 1000, (n, 2)).astype(np.float32), uid=ids)


@pytest.mark.gpu
@pytest.mark.parametrize("far", [0, 300])
@pytest.mark.parametrize("n", SIZES)
def test_sorted_ids_in_every_output(n, far):
    rng = np.random.default_rng(1000 + n)
    # ids spread over the whole int32 range, in random order
    ids = rng.choice(2**32, size=n, replace=False).astype(np.int64) - 2**31
    ids = ids.astype(np.int32)
    want = np.tile(np.sort(ids), 3)
    qs = np.zeros(3, np.int32)
    with _index(n, ids, far) as idx:
        for mode in ("fp32", "fp64"):
            # page-locked output: staged on the first call, written by the
            # kernels on the later ones
            for _ in range(3):
                got, off = idx.query_batch_flat(qs, 2, mode)
                assert np.array_equal(off, n * np.arange(4))
                assert np.array_equal(got, want)
            # pageable output
            for got in idx.query_batch(qs, 2, mode):
                assert np.array_equal(got, want[:n])
            assert np.array_equal(idx.query(0, 2, mode), want[:n])


@pytest.mark.gpu
@pytest.mark.parametrize("nq", [1023, 1024, 1025, 2049, 4097])
def test_regions_past_the_pool(nq):
    """Every query returns 9001 ids: more than a fresh workspace's pool (4096 a
    query) holds, so the first launch skips the slots past its end and the
    batch runs again; the scans' blocks take 1024 slots each."""
    n = 9001
    ids = np.random.default_rng(nq).permutation(n).astype(np.int32)
    with _index(n, ids, 0) as idx:
        for mode in ("fp64", "fp32"):
            got, off = idx.query_batch_flat(np.zeros(nq, np.int32), 3, mode)
            assert np.array_equal(off, n * np.arange(nq + 1))
            assert np.array_equal(got.reshape(nq, n), np.tile(np.arange(n, dtype=np.int32), (nq, 1)))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [513, 5000, 12_288, 16_384, 16_385])
@pytest.mark.parametrize("kind", ["even", "groups", "equal", "pairs", "two ends"])
def test_ids_in_groups(n, kind):
    """Ids spread evenly, in narrow groups (a part of their range holds many),
    all the same, each twice, and at both ends of the int32 range."""
    rng = np.random.default_rng(n)
    i = np.arange(n, dtype=np.int64)
    ids = {"even": i * 37 - 1000, "groups": (i // 200) * 1_000_003 + i % 200, "equal": np.full(n, -7, np.int64),
           "pairs": (i // 2) * 101, "two ends": np.where(i % 2 == 0, -2**31 + i, 2**31 - 1 - i)}[kind]
    ids = rng.permutation(ids).astype(np.int32)
    qs = np.zeros(3, np.int32)
    with _index(n, ids, 0) as idx:
        for mode in ("fp32", "fp64"):
            for _ in range(2):
                got, off = idx.query_batch_flat(qs, 2, mode)
                assert np.array_equal(off, n * np.arange(4))
                assert np.array_equal(got, np.tile(np.sort(ids), 3))
