"""The binding's native calls against the same calls through ctypes: results,
errors and the state after a close, with and without the built module."""
import numpy as np
import pytest

import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("native", [True, False])
def test_calls_agree(engine, monkeypatch, native):
    if not native:
        monkeypatch.setattr(engine, "_fast", False)
    ds = datagen.uniform(2000, 20_000, seed=95, nq=40, k=6)
    with engine.Index.of(ds) as idx:
        want = idx.query_batch(ds.queries, 6)
        for q, w in zip(ds.queries, want):
            for mode in ("fp64", "fp32"):
                got = idx.query(q, 6, mode)
                assert got.dtype == np.int32 and got.flags.owndata and np.array_equal(got, w)
        ids, st = idx.query(int(ds.queries[0]), 6, stats=True)
        assert np.array_equal(ids, want[0]) and st["results"] == want[0].size
        for bad in ((-1, 6), (ds.nf, 6), (0, 0)):
            with pytest.raises(engine.RkNNError) as e:
                idx.query(*bad)
            assert e.value.status == 1
        with engine.Server(idx) as srv:
            tickets = [srv.submit(q, 6) for q in ds.queries]
            for t, w in zip(tickets, want):
                assert np.array_equal(srv.wait(t), w)
            t = srv.submit(ds.queries[1], 200)          # more ids than wait's first buffer holds
            ids, ms = srv.wait(t, latency=True)
            assert ids.size > 1024 and ms > 0 and np.array_equal(ids, idx.query(ds.queries[1], 200, "fp32"))
            with pytest.raises(engine.RkNNError):
                srv.wait(t)                             # released
            with pytest.raises(engine.RkNNError):
                srv.submit(-1, 6)
        with pytest.raises(engine.RkNNError):
            srv.submit(0, 6)                            # stopped
    with pytest.raises(engine.RkNNError) as e:
        idx.query(0, 6)                                 # closed
    assert e.value.status == 1


@pytest.mark.parametrize("nq,kmax", [(1, 9), (300, 40), (300, 3000), (5000, 90)])
def test_orders_of_k(engine, nq, kmax):
    """Mixed k in one batch, where the k are counted and where they are sorted:
    the same sets as a query alone."""
    ds = datagen.uniform(3000, 15_000, seed=96, nq=50, k=1)
    rng = np.random.default_rng(nq)
    qs = rng.choice(ds.queries, nq).astype(np.int32)
    ks = rng.integers(1, kmax + 1, nq).astype(np.int32)
    with engine.Index.of(ds) as idx:
        got = idx.query_batch(qs, ks)
        for i in rng.choice(nq, min(nq, 25), replace=False):
            assert np.array_equal(got[i], idx.query(int(qs[i]), int(ks[i]), "fp32")), (int(qs[i]), int(ks[i]))
