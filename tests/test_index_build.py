"""Index creation: the points' bounding box, refused coordinates, and the
points and ids given back by a snapshot."""
import numpy as np
import pytest

import datagen
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,nu", [(1, 0), (1, 1), (31, 33), (256, 255), (257, 1_000_003)])
def test_bounding_box(engine, nf, nu):
    rng = np.random.default_rng(nf + nu)
    fxy = rng.normal(scale=300.0, size=(nf, 2)).astype(np.float32)
    uxy = (rng.normal(scale=400.0, size=(nu, 2)) - 1000.0).astype(np.float32)
    if nu:
        uxy[rng.integers(nu)] = (-0.0, 5e-42)       # signed zero, a subnormal
        uxy[-1] = (3e7, -3e7)                       # the last point decides two sides
    allp = np.concatenate([fxy, uxy])
    with engine.Index(fxy, uxy) as idx:
        inf = idx.info()
    assert [inf["x0"], inf["y0"]] == allp.min(0).tolist()
    assert [inf["x1"], inf["y1"]] == allp.max(0).tolist()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("what", ["facility", "user"])
def test_non_finite_coordinates_are_refused(engine, bad, what):
    fxy = np.ones((1000, 2), np.float32)
    uxy = np.full((5001, 2), 2.0, np.float32)
    (fxy if what == "facility" else uxy)[-1, 1] = bad
    with pytest.raises(engine.RkNNError) as e:
        engine.Index(fxy, uxy)
    assert e.value.status == 1 and what in str(e.value)


@pytest.mark.parametrize("given", [True, False])
def test_snapshot_keeps_points_and_ids(engine, tmp_path, given):
    rng = np.random.default_rng(5)
    fxy = rng.uniform(size=(513, 2)).astype(np.float32)
    uxy = rng.uniform(size=(2049, 2)).astype(np.float32)
    fid = rng.permutation(513).astype(np.int32) if given else None
    path = str(tmp_path / "a.rkx")
    with engine.Index(fxy, uxy, fid=fid) as idx:
        idx.save(path)
        want_uid = idx.uid
    f, i, u, j = engine.snapshot_read(path)
    assert np.array_equal(f, fxy) and np.array_equal(u, uxy) and np.array_equal(j, want_uid)
    assert np.array_equal(i, fid if given else np.arange(513))


@pytest.mark.parametrize("nu", [1, 255, 2047, 2048, 2049, 70_001])
@pytest.mark.parametrize("per_cell", [1e9, 300.0, 4.0, 1e-6])
def test_cells(engine, nu, per_cell):
    """Sort passes (1 to 4 digits: one cell, and up to 8192 x 8192), tiles'
    remainders, cells of many users and none: the answers are the oracle's."""
    rng = np.random.default_rng(nu)
    uxy = rng.uniform(0, 1000, size=(nu, 2))
    uxy[: nu // 2] = np.round(uxy[: nu // 2] / 250) * 250       # half in crowded points
    fxy = rng.uniform(0, 1000, size=(400, 2)).astype(np.float32)
    fxy[:40] = fxy[0]                                           # coincident facilities
    ds = datagen.Dataset(fxy, uxy.astype(np.float32), np.arange(400, dtype=np.int32),
                         np.arange(400, 400 + nu, dtype=np.int32), np.arange(0, 400, 37).astype(np.int64))
    o = O.Oracle.of(ds)
    with engine.Index.of(ds, usr_per_cell=per_cell, fac_per_cell=min(per_cell, 1e3)) as idx:
        for k in (1, 9):
            want = [o.query(int(q), k) for q in ds.queries]
            for got, w in zip(idx.query_batch(ds.queries, k, "fp32"), want):
                assert np.array_equal(got, w), (nu, per_cell, k)
