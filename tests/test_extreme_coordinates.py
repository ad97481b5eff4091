"""Coordinates near the ends of the float range, which an index accepts like any
others: sums and squares of offsets overflow or lose their accuracy there, and
the certified float tests have to leave such pairs to the exact count.  Results
are id sets: equality is bit-exact."""
import numpy as np
import pytest

import datagen
import oracle as O

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


def _points(layout):
    """Points on multiples of 2^-23, so that scaling them by a power of two is
    exact and changes no result: the unscaled set is the oracle's."""
    rng = np.random.default_rng(3)
    if layout == "far":                     # users around few facilities, up to three times as far out
        f, u = 1.3 * rng.random((30, 2)) - 0.65, 3.2 * rng.random((3000, 2)) - 1.6
    elif layout == "clustered":
        c = rng.random((20, 2))
        f = c[rng.integers(20, size=1500)] + 0.01 * rng.standard_normal((1500, 2))
        u = c[rng.integers(20, size=3000)] + 0.02 * rng.standard_normal((3000, 2))
    else:
        f, u = rng.random((600, 2)) - 0.5, rng.random((3000, 2)) - 0.5
    return (np.round(v * 2.0**23) / 2.0**23 for v in (f, u))


@pytest.fixture(scope="module", params=["centred", "clustered", "far"])
def points(request):
    f, u = _points(request.param)
    o = O.Oracle.of(_set(f, u))
    qs = np.random.default_rng(1).integers(0, len(f), 40).astype(np.int32)
    ks = (1, 3, 8) if request.param == "far" else (1, 10, 40)
    return f, u, qs, {k: [o.query(int(q), k) for q in qs] for k in ks}


def _check(engine, points, e, filter, modes, sizes):
    f, u, qs, want = points
    with engine.Index.of(_set(f * 2.0**e, u * 2.0**e), filter=filter) as idx:
        for mode in modes:
            for k, w in want.items():
                if filter == "inf" and k > 10:
                    continue
                for n in sizes:
                    got = idx.query_batch(np.resize(qs, n), k, mode)
                    bad = [i for i, g in enumerate(got) if not np.array_equal(g, w[i % len(qs)])]
                    assert not bad, (e, filter, mode, k, n, len(bad))


@pytest.mark.parametrize("e", [-90, -72, -66, 64, 66, 90])
def test_scaled_points_zone_fp64(engine, points, e):
    """Through the zone, whose candidates the exact count decides: listed whole
    in small batches, behind the boxes in larger ones."""
    _check(engine, points, e, "inf", ("fp64",), (1, 40))


@pytest.mark.parametrize("e,modes", [(-90, ("fp32", "fp64")), (-72, ("fp32", "fp64")), (-66, ("fp32", "fp64")),
                                     (64, ("fp64",)), (66, ("fp64",)), (90, ("fp64",))])
def test_scaled_points_slice(engine, points, e, modes):
    """Through the slice filter, two warps a query and one."""
    _check(engine, points, e, "slice", modes, (1, 40, 1400))


@pytest.mark.parametrize("filter", ["slice", "inf"])
@pytest.mark.parametrize("e", [64, 66, 90])
def test_scaled_points_fp32(engine, points, e, filter):
    """Float evaluations that overflow decide nothing, user by user (in the
    filter's own blocks and in the verification kernel) and behind boxes."""
    _check(engine, points, e, filter, ("fp32",), (1, 40) if filter == "inf" else (1, 40, 1400))
