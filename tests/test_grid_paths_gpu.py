"""Sizes around the lines between the grid builds (one block up to 4096 points
and 4096 cells) and between the tile-table builds (one block up to 32 cells per
side): each build holds the same cells, and the counts over its tiles are the
brute force's."""
import numpy as np
import pytest

import oracle
from desi_b200 import catalog
from desi_b200._lib import PCF_OPT_GRID_BUILD

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("source", ["host", "device"])
@pytest.mark.parametrize("weights", ["unit", "uniform"])
@pytest.mark.parametrize("n,P", [(1, 1), (2, 16), (3, 2), (31, 16), (33, 4), (1023, 16), (1024, 15), (1025, 17),
                                 (4091, 16), (4095, 16), (4096, 16), (4097, 16), (4096, 17), (3000, 32), (3000, 33),
                                 (3000, 65)])
def test_cells_and_tiles(ctx, n, P, weights, source):
    pts = catalog.neyman_scott(n, 100.0, seed=n + P, children=20, weights=weights)
    other = catalog.uniform(257, 100.0, seed=7, weights=weights)
    if source == "device":
        import torch

        dev = torch.from_numpy(pts).cuda()
        torch.cuda.synchronize()
        g = ctx.grid(None, 100.0, partitions=P, device_ptr=dev.data_ptr(), n=n)
    else:
        g = ctx.grid(pts, 100.0, partitions=P)
    ctx.set_option(PCF_OPT_GRID_BUILD, 1)
    ref = ctx.grid(pts, 100.0, partitions=P)
    ctx.set_option(PCF_OPT_GRID_BUILD, 0)
    (p, start), (q, want) = g.download(), ref.download()
    np.testing.assert_array_equal(start, want)
    cell = np.repeat(np.arange(P ** 3), np.diff(start))
    order = lambda a: a[np.lexsort((a[:, 3], a[:, 2], a[:, 1], a[:, 0], cell))]  # noqa: E731
    np.testing.assert_array_equal(order(p), order(q))
    assert g.info()["nonempty_cells"] == ref.info()["nonempty_cells"] == np.count_nonzero(np.diff(start))
    o = ctx.grid(other, 100.0, partitions=P)
    got = ctx.count_pairs(g, o, bins=7, dmax=11.0)
    exp = oracle.pairs(pts, other, box=100.0, bins=7, dmax=11.0, ani=False, bpc=False)
    np.testing.assert_allclose(got, exp, rtol=0 if weights == "unit" else 1e-12, atol=0)


def test_point_outside_the_box(ctx):
    for n in (5, 5000):
        pts = catalog.uniform(n, 100.0, seed=1)
        pts[n // 2, 1] = 100.0
        with pytest.raises(Exception, match="outside"):
            ctx.grid(pts, 100.0)
