"""Node-gated isotropic counts as corrections of the plain ones: node grids with
dmax a whole number of nodes, a diagonal that touches the gate's bound (which
takes every ordered triangle), coarse and fine nodes, and catalogs of a few
points, against the oracle; and larger ones against the general path, which a
catalog of weight 1/2 takes (its sums are the counts / 8, exactly)."""

import numpy as np
import pytest

import oracle
from desi_b200 import catalog

pytestmark = pytest.mark.gpu


def both(n, m, box, seed):
    return catalog.neyman_scott(n, box, seed=seed, children=max(2, n // 8)), catalog.uniform(m, box, seed=seed + 1)


@pytest.mark.parametrize("n,m,box,P,dmax,bins", [
    (1, 2, 100.0, 10, 30.0, 5), (3, 2, 100.0, 5, 49.0, 4), (40, 33, 100.0, 10, 30.0, 7),
    (300, 250, 100.0, 3, 45.0, 9), (300, 250, 100.0, 25, 20.0, 6), (300, 250, 250.0, 35, 80.0, 30),
    (300, 250, 100.0, 4, 43.30127, 8), (300, 250, 100.0, 10, 34.641016, 8), (200, 300, 100.0, 200, 33.3, 255),
    (300, 250, 100.0, 1, 40.0, 5)])
def test_against_the_oracle(ctx, n, m, box, P, dmax, bins):
    D, R = both(n, m, box, n + P)
    gd, gr = ctx.grid(D, box, partitions=P), ctx.grid(R, box, partitions=P)
    for x, y, X, Y in ((gd, None, D, None), (gr, None, R, None), (gd, gr, D, R), (gr, gd, R, D)):
        got, st = ctx.count_triplets(x, y, bins=bins, dmax=dmax, bpc=True, ref_gates=True, stats=True)
        want = oracle.triplets_iso(X, Y, box=box, bins=bins, dmax=dmax, bpc=True, ref_gates=P)
        np.testing.assert_array_equal(got, want)
        assert st["pairs"] == want.sum()


@pytest.mark.parametrize("P,dmax", [(20, 61.7), (35, 79.9), (7, 100.0), (96, 40.0)])
def test_against_the_general_path(ctx, P, dmax):
    box, bins = 250.0, 30
    D, R = both(2500, 3600, box, P)
    half = lambda a: np.concatenate([a[:, :3], np.full((len(a), 1), 0.5, np.float32)], 1)  # noqa: E731
    gd, gr = ctx.grid(D, box, partitions=P), ctx.grid(R, box, partitions=P)
    hd, hr = ctx.grid(half(D), box, partitions=P), ctx.grid(half(R), box, partitions=P)
    kw = dict(bins=bins, dmax=dmax, bpc=True, ref_gates=True)
    for a, b, ha, hb in ((gd, None, hd, None), (gr, None, hr, None), (gd, gr, hd, hr), (gr, gd, hr, hd)):
        np.testing.assert_array_equal(ctx.count_triplets(a, b, **kw), 8.0 * ctx.count_triplets(ha, hb, **kw))
