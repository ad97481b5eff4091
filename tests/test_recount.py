"""The exact count over survivors from fewer than the GPU has warps to dozens
for each of them (groups of warps a survivor, one, runs from the queue), behind
the influence zone, which leaves about half of its candidates to it.  Results
are id sets: equality is bit-exact."""
import numpy as np
import pytest

import datagen
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def uni():
    ds = datagen.uniform(3000, 90_000, seed=75, nq=60, k=1)
    o = O.Oracle.of(ds)
    return ds, {k: [o.query(int(q), k) for q in ds.queries] for k in (2, 12)}


@pytest.mark.parametrize("mode", ["fp32", "fp64"])
@pytest.mark.parametrize("nq", [1, 9, 17, 120, 700, 3000, 20_000])
def test_counts_at_every_depth_of_the_queue(engine, uni, nq, mode):
    ds, want = uni
    with engine.Index.of(ds, filter="inf") as idx:
        for k in want:
            if nq * k > 60_000:
                continue
            got, off = idx.query_batch_flat(np.resize(ds.queries, nq).astype(np.int32), k, mode)
            for i in range(nq):
                assert np.array_equal(got[off[i]:off[i + 1]], want[k][i % 60]), (nq, k, i)
