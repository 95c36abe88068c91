"""Cells per side of counts that the general pair kernel makes (signed weights):
the histograms at the sizes where the rule changes, and that small catalogs get
cells enough to fill the device."""
import numpy as np
import pytest

import oracle
from desi_b200 import catalog

pytestmark = pytest.mark.gpu


def _signed(pts, seed):
    pts[:, 3] = np.random.default_rng(seed).uniform(-1.0, 1.0, len(pts)).astype(np.float32)
    return pts


@pytest.mark.parametrize("na,nb,dmax", [(3, 4, 40.0), (1249, 1250, 100.0), (1250, 1251, 100.0), (5000, 4000, 30.0),
                                        (50000, 20, 25.0), (50001, 20, 25.0), (3000, 50001, 6.0)])
@pytest.mark.parametrize("bpc", [False, True])
def test_values(ctx, na, nb, dmax, bpc):
    box = 250.0
    a = _signed(catalog.neyman_scott(na, box, seed=na), 1)
    b = _signed(catalog.uniform(nb, box, seed=nb), 2)
    ga, gb = ctx.grid(a, box), ctx.grid(b, box)
    a1, b1 = a.copy(), b.copy()
    a1[:, 3], b1[:, 3] = np.abs(a[:, 3]), np.abs(b[:, 3])
    for ani in (False, True):
        kw = dict(bins=9, dmax=dmax, ani=ani, bpc=bpc)
        got = ctx.count_pairs(ga, gb, **kw)
        want, size = oracle.pairs(a, b, box=box, **kw), oracle.pairs(a1, b1, box=box, **kw)
        assert np.all(np.abs(got - want) <= 1e-12 * size)


@pytest.mark.parametrize("dmax,bpc,cells", [(200.0, True, 6), (450.0, False, 8)])
def test_default_is_no_slower_than_finer_cells(ctx, dmax, bpc, cells):
    """3000 against 4000 points, whose few cells left SMs idle under the rule of the
    branch-free kernel (4 and 6 cells per side: 1.4 times the time)."""
    a = _signed(catalog.neyman_scott(3000, 1000.0, seed=3), 3)
    b = _signed(catalog.uniform(4000, 1000.0, seed=4), 4)

    def best(partitions):
        ga, gb = ctx.grid(a, 1000.0, partitions=partitions), ctx.grid(b, 1000.0, partitions=partitions)
        kw = dict(bins=30, dmax=dmax, bpc=bpc, stats=True)
        return min(ctx.count_pairs(ga, gb, **kw)[1]["kernel_ms"] for _ in range(12))

    best(0)
    assert best(0) <= 1.2 * best(cells)
