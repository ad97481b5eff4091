"""rknn_last_zone: the facilities of a slot's half-planes as input indices."""
import numpy as np
import pytest

import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,filter,k", [(1, "inf", 1), (2000, "inf", 5), (2000, "slice", 40)])
def test_facilities_of_the_last_zone(engine, nf, filter, k):
    ds = datagen.uniform(nf, 20_000, seed=72, nq=min(nf, 5), k=k)
    with engine.Index.of(ds, filter=filter) as idx:
        idx.query_batch(ds.queries, k, "fp32")
        for slot, q in enumerate(ds.queries):
            fac, _ = idx.last_zone(slot)
            assert len(set(fac.tolist())) == fac.size and q not in fac
            assert np.all((fac >= 0) & (fac < nf))
            # the nearest k + 1 facilities are among them
            d = np.sum((ds.fxy.astype(np.float64) - ds.fxy[q].astype(np.float64)) ** 2, 1)
            near = [i for i in np.argsort(d, kind="stable") if i != q][:k + 1]
            assert set(near) <= set(fac.tolist())
