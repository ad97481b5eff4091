"""The binding's native module: built and loaded wherever the interpreter's
headers are installed, with every entry point that rknn.py calls, so that the
native half of the binding's tests does not run through ctypes unnoticed."""
import os
import sysconfig

import numpy as np
import pytest

import datagen

HEADERS = os.path.exists(os.path.join(sysconfig.get_paths().get("include") or "", "Python.h"))
NAMES = ("query_batch", "query", "serve_submit", "serve_wait")


@pytest.mark.skipif(not HEADERS, reason="the interpreter's headers are not installed")
def test_module_is_loaded(engine):
    fast = engine._fast_call()
    assert fast, "built beside the library but not importable"
    assert all(callable(getattr(fast, n, None)) for n in NAMES)


@pytest.mark.gpu
@pytest.mark.skipif(not HEADERS, reason="the interpreter's headers are not installed")
def test_calls_take_the_module(engine, monkeypatch):
    """Each call of the binding reaches its native entry point."""
    fast, seen = engine._fast_call(), set()

    class Spy:
        def __getattr__(self, name):
            seen.add(name)
            return getattr(fast, name)

    monkeypatch.setattr(engine, "_fast", Spy())
    ds = datagen.uniform(500, 4000, seed=77, nq=5, k=3)
    with engine.Index.of(ds) as idx:
        want = idx.query(int(ds.queries[0]), 3)
        got, off = idx.query_batch_flat(ds.queries.astype(np.int32), 3)
        assert np.array_equal(got[:off[1]], want)
        with engine.Server(idx) as srv:
            assert np.array_equal(srv.wait(srv.submit(int(ds.queries[0]), 3)), want)
    assert seen == set(NAMES)
