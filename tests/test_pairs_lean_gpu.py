"""Sizes at which the branch-free pair kernel can go wrong: ranges around its
candidate windows (32) and steps, home tiles of few points (several candidate
streams), bin counts around its readout and column choices, counters whose
upper limbs carry, and batches whose jobs are smaller than a CTA's items."""
import numpy as np
import pytest

import oracle
from desi_b200 import catalog

pytestmark = pytest.mark.gpu


def check(ctx, a, b, box, bins, dmax, bpc, weighted, **grid):
    ga, gb = ctx.grid(a, box, **grid), ctx.grid(b, box, **grid)
    for x, y, X, Y in ((ga, None, a, None), (ga, gb, a, b)):
        want = [oracle.pairs(X, Y, box=box, bins=bins, dmax=dmax, ani=k, bpc=bpc) for k in (False, True)]
        got = [ctx.count_pairs(x, y, bins=bins, dmax=dmax, ani=k, bpc=bpc) for k in (False, True)]
        got += ctx.count_pairs(x, y, bins=bins, dmax=dmax, ani="both", bpc=bpc)
        for g, w in zip(got, want + want):
            if weighted:  # integer weight products are exact: only the final sums round
                np.testing.assert_allclose(g, w, rtol=1e-12, atol=0)
            else:
                np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("weights", ["unit", "uniform"])
@pytest.mark.parametrize("na,nb,partitions", [(1, 1, 0), (2, 3, 7), (31, 33, 0), (64, 65, 0), (97, 200, 5),
                                              (300, 1, 9), (700, 513, 20)])
@pytest.mark.parametrize("bpc", [False, True])
def test_sizes(ctx, na, nb, partitions, weights, bpc):
    a = catalog.neyman_scott(na, 100.0, seed=na, children=40, weights=weights)
    b = catalog.uniform(nb, 100.0, seed=nb + 1, weights=weights)
    check(ctx, a, b, 100.0, 17, 33.0, bpc, weights != "unit", partitions=partitions)


@pytest.mark.parametrize("weights", ["unit", "uniform"])
@pytest.mark.parametrize("bins", [1, 2, 46, 47, 60, 92, 93, 119, 120, 121, 126, 200, 255, 256])
def test_bin_counts(ctx, bins, weights):
    a = catalog.neyman_scott(500, 100.0, seed=5, weights=weights)
    b = catalog.uniform(400, 100.0, seed=6, weights=weights)
    check(ctx, a, b, 100.0, bins, 40.0, True, weights != "unit")


@pytest.mark.parametrize("dmax", [230.7, 700.3, 30000.7])
def test_large_dmax(ctx, dmax):
    """The last bin's edge lies up to dmax * 1e-6 bins beyond dmax."""
    box = 3.4 * dmax
    for w in ("unit", "uniform"):
        check(ctx, catalog.uniform(900, box, seed=11, weights=w), catalog.uniform(800, box, seed=12, weights=w), box,
              13, dmax, True, w != "unit")


@pytest.mark.parametrize("spread", [0.3, 0.003])
def test_limbs_carry(ctx, spread):
    """A clump whose pairs share a few bins: the second limb of a weighted
    counter overflows many times over (at 16384 adds)."""
    rng = np.random.default_rng(9)

    def clump(n):
        p = np.empty((n, 4), np.float32)
        p[:, :3] = 50.0 + rng.normal(0.0, spread, (n, 3))
        p[:, 3] = rng.uniform(1.4, 1.9999, n)
        return p

    check(ctx, clump(2500), clump(2300), 100.0, 12, 24.0, False, True)


def test_batch_of_small_jobs(ctx):
    D = catalog.neyman_scott(900, 200.0, seed=1, weights="uniform")
    Rs = [catalog.uniform(n, 200.0, seed=10 + n, weights="uniform") for n in (1, 700, 2, 40, 5, 1500, 3, 3, 90)]
    gd, gr = ctx.grid(D, 200.0), [ctx.grid(R, 200.0) for R in Rs]
    for ani in (False, True):
        dd, rr, dr = ctx.batch_pairs(gd, gr, bins=15, dmax=50.0, ani=ani, bpc=True)
        kw = dict(box=200.0, bins=15, dmax=50.0, ani=ani, bpc=True)
        np.testing.assert_allclose(dd, oracle.pairs(D, None, **kw), rtol=1e-12, atol=0)
        for i, R in enumerate(Rs):
            np.testing.assert_allclose(rr[i], oracle.pairs(R, None, **kw), rtol=1e-12, atol=0)
            np.testing.assert_allclose(dr[i], oracle.pairs(D, R, **kw), rtol=1e-12, atol=0)
