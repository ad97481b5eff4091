"""Coordinates near the ends of the float range, which an index accepts like any
others: sums and squares of offsets overflow or lose their accuracy there, and
the certified float tests have to leave such pairs to the exact count.  Results
are id sets: equality is bit-exact."""
import numpy as np
import pytest

import datagen

pytestmark = pytest.mark.gpu


def _set(fxy, uxy):
    nf, nu = len(fxy), len(uxy)
    return datagen.Dataset(np.asarray(fxy, np.float32), np.asarray(uxy, np.float32), np.arange(nf, dtype=np.int32),
                           np.arange(nf, nf + nu, dtype=np.int32))


def test_half_plane_overflows_on_the_way(engine):
    """b y + c of the half-plane's value overflows for this user, the value
    itself (9.6e37: q is nearer) does not."""
    ds = _set([[0, 0], [1.2e19, 1.2e19]], [[-2.1e19, 2.9e19]])
    f, u = ds.fxy.astype(np.float64), ds.uxy[0].astype(np.float64)
    assert np.sum((u - f[0]) ** 2) < np.sum((u - f[1]) ** 2)
    with engine.Index.of(ds, filter="slice") as idx:
        assert idx.query(0, 1, "fp64").tolist() == [2]
