"""Index creation: the points' bounding box, refused coordinates, and the
points and ids given back by a snapshot."""
import numpy as np
import pytest

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
