"""Tuning that fails on the way (the workspace's sizing, made to fail on the
host: no GPU fault): the index keeps the densities and the verification shape
it had, and answers as before."""
import ctypes as C

import numpy as np
import pytest

import datagen

pytestmark = pytest.mark.gpu

# sizings of the workspace: two a query call, three calls a trial; a trial on
# entry, 25 of densities, then 9 of shapes
TRIAL = 6


def _shape(lib, idx):
    out = (C.c_int32 * 3)()
    assert lib.rknn_debug_shape(idx.h, out) == 0
    return list(out)


@pytest.mark.parametrize("opts", [{}, {"users_per_thread": 8, "verify_warps": 16}])
@pytest.mark.parametrize("trial", [0, 1, 13, 26, 30, 34])
def test_failed_tuning_changes_nothing(engine, opts, trial):
    lib = engine.load()
    ds = datagen.uniform(2000, 20_000, seed=71, nq=40, k=5)
    with engine.Index.of(ds, **opts) as idx:
        info, shape = idx.info(), _shape(lib, idx)
        want = [idx.query_batch(ds.queries, 5, m) for m in ("fp32", "fp64")]
        assert lib.rknn_debug_fail_workspace(idx.h, TRIAL * trial + 3) == 0
        with pytest.raises(engine.RkNNError) as e:
            idx.tune(ds.queries, 5, "fp64")
        assert e.value.status == 2
        assert idx.info() == info and _shape(lib, idx) == shape
        for m, w in zip(("fp32", "fp64"), want):
            assert all(np.array_equal(a, b) for a, b in zip(idx.query_batch(ds.queries, 5, m), w))
        assert idx.tune(ds.queries, 5, "fp64")["trials"] == 34
