"""The slice filter's kept region as user-grid rows: regions of more rows than
it lists one by one, regions cut by the data's box, points on a line, users far
from every facility, more facilities in a cell than half-planes are kept.  Every answer equals the exact oracle's."""
import numpy as np
import pytest

import datagen
import oracle as O

pytestmark = pytest.mark.gpu


def _points(layout):
    rng = np.random.default_rng(91)
    if layout == "wide":                    # about 190 user rows, regions from a few to all of them
        f, u = rng.uniform(0, 1000, (60, 2)), rng.uniform(0, 1000, (300_007, 2))
    elif layout == "vertical":              # one column of cells
        f = np.stack([np.full(200, 3.0), rng.uniform(-50, 50, 200)], 1)
        u = np.stack([np.full(20_011, 3.0), rng.uniform(-50, 50, 20_011)], 1)
    elif layout == "horizontal":
        f = np.stack([rng.uniform(-50, 50, 200), np.full(200, -7.0)], 1)
        u = np.stack([rng.uniform(-50, 50, 20_011), np.full(20_011, -7.0)], 1)
    elif layout == "dense":                 # cells of thousands of facilities beside empty ones
        f = np.concatenate([rng.normal((400, 400), 0.3, (4000, 2)), rng.uniform(0, 1000, (400, 2))])
        u = np.concatenate([rng.normal((400, 400), 0.4, (8000, 2)), rng.uniform(0, 1000, (30_000, 2))])
    else:                                   # users in a corner, facilities in the opposite one
        f = rng.uniform(0, 10, (150, 2))
        u = np.concatenate([rng.uniform(900, 1000, (30_000, 2)), rng.uniform(0, 10, (500, 2))])
    f, u = f.astype(np.float32), u.astype(np.float32)
    return datagen.Dataset(f, u, np.arange(len(f), dtype=np.int32), np.arange(len(f), len(f) + len(u), dtype=np.int32))


@pytest.mark.parametrize("layout", ["wide", "vertical", "horizontal", "dense", "corner"])
def test_regions_match_oracle(engine, layout):
    ds = _points(layout)
    o = O.Oracle.of(ds)
    # the facilities nearest to the box's sides and corners, and a few others
    near = [np.argmin(ds.fxy @ np.array(d, np.float32)) for d in [(1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, -1)]]
    qs = np.unique(np.concatenate([near, np.arange(0, ds.nf, max(9, ds.nf // 25))])).astype(np.int32)
    big = np.tile(qs, 1 + 1300 // qs.size)          # one warp a query instead of two
    with engine.Index.of(ds, filter="slice") as idx:
        for k in (1, 7, 20, 45):
            want = [o.query(int(q), k) for q in qs]
            for mode in ("fp32", "fp64"):
                for got, w in zip(idx.query_batch(qs, k, mode), want):
                    assert np.array_equal(got, w), (layout, k, mode)
            if layout != "corner":
                for got, w in zip(idx.query_batch(big, k, "fp32"), want * (big.size // qs.size)):
                    assert np.array_equal(got, w), (layout, k)


@pytest.mark.parametrize("spread", [0.2, 3.0, 14.0, 25.0, 300.0])
def test_clustered_facilities(engine, spread):
    """Facility grids from nearly empty to uniformly filled: small batches take
    one warp a query below half the uniform filling, two above."""
    rng = np.random.default_rng(int(10 * spread))
    centre = rng.uniform(0, 1000, (60, 2))
    f = centre[rng.integers(60, size=12_000)] + spread * rng.standard_normal((12_000, 2))
    u = np.concatenate([centre[rng.integers(60, size=30_000)] + 2 * spread * rng.standard_normal((30_000, 2)),
                        rng.uniform(0, 1000, (10_000, 2))])
    f, u = f.astype(np.float32), u.astype(np.float32)
    ds = datagen.Dataset(f, u, np.arange(12_000, dtype=np.int32), np.arange(12_000, 52_000, dtype=np.int32))
    o = O.Oracle.of(ds)
    qs = np.arange(0, 12_000, 299, dtype=np.int32)
    with engine.Index.of(ds) as idx:
        for k in (1, 10, 31):
            want = [o.query(int(q), k) for q in qs]
            for mode in ("fp32", "fp64"):
                for n in (1, qs.size):
                    for got, w in zip(idx.query_batch(qs[:n], k, mode), want):
                        assert np.array_equal(got, w), (spread, k, mode, n)
