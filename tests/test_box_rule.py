"""FP32 slots on either side of the line from which boxes come before the
user-by-user test (k (n - 750) against 16 n for n candidates), beside slots of
the other kind in one batch, against the exact oracle.  Results are id sets:
equality is bit-exact."""
import numpy as np
import pytest

import datagen
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,nu,ks", [
    (3000, 30_011, (16, 40, 60, 64, 68, 72, 80, 100)),      # about 14 candidates for each of k: the line near k = 70
    (400, 30_011, (7, 15, 16, 17, 20, 24, 28, 40)),         # about 100: near k = 22
])
def test_both_sides_of_the_line(engine, nf, nu, ks):
    ds = datagen.uniform(nf, nu, seed=74, nq=30, k=1)
    o = O.Oracle.of(ds)
    want = {(int(q), k): o.query(int(q), k) for q in ds.queries for k in ks}
    rng = np.random.default_rng(nf)
    with engine.Index.of(ds, filter="slice") as idx:
        for n in (17, 1500):                # above k = 32 and in larger batches the verification kernel's slots
            qs = rng.choice(ds.queries, n).astype(np.int32)
            for mixed in (False, True):
                for k in (ks[:1] if mixed else ks):
                    kk = rng.choice(ks, n).astype(np.int32) if mixed else np.full(n, k, np.int32)
                    for q, k1, got in zip(qs, kk, idx.query_batch(qs, kk, "fp32")):
                        assert np.array_equal(got, want[(int(q), int(k1))]), (int(q), int(k1), n)


@pytest.mark.parametrize("nq", [7295, 7296, 14_591, 14_592])
def test_parts_of_an_item(engine, nq):
    """Items of one, two and four parts on either side of where the queries
    outnumber the resident warps (3,648 at these half-planes) two and four times."""
    ds = datagen.uniform(900, 30_011, seed=76, nq=40, k=1)
    o = O.Oracle.of(ds)
    want = {k: [o.query(int(q), k) for q in ds.queries] for k in (2, 9, 35)}
    with engine.Index.of(ds) as idx:
        for k, w in want.items():
            for mode in ("fp32", "fp64"):
                got, off = idx.query_batch_flat(np.resize(ds.queries, nq).astype(np.int32), k, mode)
                assert np.array_equal(np.diff(off), np.resize([x.size for x in w], nq)), (nq, k, mode)
                for i in [*range(40), *range(nq - 40, nq)]:
                    assert np.array_equal(got[off[i]:off[i + 1]], w[i % 40]), (nq, k, mode, i)
