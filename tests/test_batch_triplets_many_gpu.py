"""A triplet batch takes any number of random catalogs (600 jobs here)."""
import numpy as np
import pytest

import oracle
from desi_b200 import catalog

pytestmark = pytest.mark.gpu


def test_two_hundred_catalogs(ctx):
    box, bins, dmax, nr = 100.0, 4, 20.0, 200
    D = catalog.neyman_scott(120, box, seed=1)
    Rs = [catalog.uniform(40 + i % 7, box, seed=10 + i) for i in range(nr)]
    gd, grs = ctx.grid(D, box), [ctx.grid(R, box) for R in Rs]
    ddd, rrr, ddr, drr = ctx.batch_triplets(gd, grs, bins=bins, dmax=dmax, bpc=True)
    kw = dict(box=box, bins=bins, dmax=dmax, bpc=True)
    np.testing.assert_array_equal(ddd, oracle.triplets_iso(D, **kw))
    for i in (0, 1, 77, 198, 199):
        np.testing.assert_array_equal(rrr[i], oracle.triplets_iso(Rs[i], **kw))
        np.testing.assert_array_equal(ddr[i], oracle.triplets_iso(D, Rs[i], **kw))
        np.testing.assert_array_equal(drr[i], oracle.triplets_iso(Rs[i], D, **kw))
