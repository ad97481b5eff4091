"""The box-first verification against the exact oracle, where it can go wrong:
candidate counts on either side of the rule that chooses it, item and group
remainders, users on a lattice (boxes of no extent, exact ties on bisectors),
every work-item shape, batches large enough for several parts an item.
Results are id sets: equality is bit-exact."""
import numpy as np
import pytest

import datagen
import oracle as O

pytestmark = pytest.mark.gpu


def _lattice(nf, nu, seed):
    """Facilities and users on a coarse integer lattice: many users share a
    point, many lie exactly on bisectors or on facilities."""
    rng = np.random.default_rng(seed)
    f = rng.choice(120 * 120, size=nf, replace=False)
    fxy = np.stack([f % 120, f // 120], 1).astype(np.float32) * 8
    uxy = rng.integers(0, 240, size=(nu, 2)).astype(np.float32) * 4
    return datagen.Dataset(fxy, uxy, np.arange(nf, dtype=np.int32), np.arange(nf, nf + nu, dtype=np.int32),
                           rng.choice(nf, size=24, replace=False).astype(np.int64))


@pytest.fixture(scope="module")
def sets():
    out = {"uniform": datagen.uniform(500, 33_333, seed=81, nq=24, k=1), "lattice": _lattice(600, 30_011, 82),
           "street": datagen.street(nu=40_009, nf=400, seed=83, nq=24, side=40, jitter=0.5)}
    return {n: (ds, O.Oracle.of(ds)) for n, ds in out.items()}


@pytest.mark.parametrize("layout", ["uniform", "lattice", "street"])
@pytest.mark.parametrize("upt,warps", [(0, 0), (2, 4), (8, 16)])
def test_boxes_match_oracle(engine, sets, layout, upt, warps):
    ds, o = sets[layout]
    with engine.Index.of(ds, users_per_thread=upt, verify_warps=warps) as idx:
        # about 66 users a facility: 5 to 8 and 33 to 100 lie on either side
        # of the rule
        for k in (1, 5, 7, 8, 33, 100, 130):
            want = [o.query(int(q), k) for q in ds.queries]
            for mode in ("fp32", "fp64"):
                for n in (len(ds.queries), 3):
                    for got, w in zip(idx.query_batch(ds.queries[:n], k, mode), want):
                        assert np.array_equal(got, w), (layout, k, mode, n)


@pytest.mark.parametrize("nq", [8192, 16_400])
def test_items_of_several_parts(engine, sets, nq):
    ds, o = sets["street"]
    rng = np.random.default_rng(nq)
    qs = rng.choice(ds.queries, size=nq).astype(np.int32)
    ks = rng.choice([1, 6, 31], size=nq).astype(np.int32)
    want = {(int(q), int(k)): o.query(int(q), int(k)) for q in ds.queries for k in (1, 6, 31)}
    with engine.Index.of(ds) as idx:
        for mode in ("fp32", "fp64"):
            for q, k, got in zip(qs, ks, idx.query_batch(qs, ks, mode)):
                assert np.array_equal(got, want[(int(q), int(k))]), (int(q), int(k), mode)


@pytest.mark.parametrize("tight", [0.0, 0.3, 0.9])
def test_quarters(engine, tight):
    """Users in clumps of eight, some of no extent, some wide: of a group's
    quarters one, two or more stay open after the boxes."""
    rng = np.random.default_rng(int(100 * tight) + 5)
    nc, nf = 4_003, 300
    centre = rng.random((nc, 1, 2)) * 1000
    wide = np.where(rng.random((nc, 1, 1)) < tight, 0.0, rng.choice([0.5, 8.0, 40.0], size=(nc, 1, 1)))
    uxy = (centre + wide * rng.standard_normal((nc, 8, 2))).reshape(-1, 2).astype(np.float32)
    fxy = (rng.random((nf, 2)) * 1000).astype(np.float32)
    ds = datagen.Dataset(fxy, uxy, np.arange(nf, dtype=np.int32), np.arange(nf, nf + 8 * nc, dtype=np.int32),
                         rng.choice(nf, size=12, replace=False).astype(np.int64))
    o = O.Oracle.of(ds)
    with engine.Index.of(ds) as idx:
        for k in (6, 17, 60):
            want = [o.query(int(q), k) for q in ds.queries]
            for mode in ("fp32", "fp64"):
                for got, w in zip(idx.query_batch(ds.queries, k, mode), want):
                    assert np.array_equal(got, w), (tight, k, mode)
