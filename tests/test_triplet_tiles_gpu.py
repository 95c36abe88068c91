"""Sizes at which the tiled unit-weight triplet counts can go wrong: lists
around the tile (8) and chunk (32) sizes, lists beyond shared memory, dmax
far from the last bin's edge, more stencil rows than one row table holds."""
import numpy as np
import pytest

import oracle
from desi_b200 import catalog

pytestmark = pytest.mark.gpu


def check(ctx, x, y, box, bins, dmax, bpc, partitions=0):
    gx = ctx.grid(x, box, partitions=partitions)
    gy = ctx.grid(y, box, partitions=partitions)
    for a, b, A, B in ((gx, None, x, None), (gx, gy, x, y), (gy, gx, y, x)):
        got, st = ctx.count_triplets(a, b, bins=bins, dmax=dmax, bpc=bpc, stats=True)
        want = oracle.triplets_iso(A, B, box=box, bins=bins, dmax=dmax, bpc=bpc)
        np.testing.assert_array_equal(got, want)
        # the reported triangles: each is in the histogram 6 times (XXX) or 2 (XXY)
        assert st["pairs"] == want.sum() / (6 if B is None else 2)


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 31), (3, 32), (8, 33), (9, 7), (10, 64), (33, 65), (34, 1), (65, 130)])
def test_list_sizes(ctx, nx, ny):
    rng = np.random.default_rng(nx * 100 + ny)

    def clump(n):  # every point within dmax of every other: lists hold n or n - 1 - i entries
        return np.concatenate([rng.uniform(45.0, 60.0, (n, 3)), np.ones((n, 1))], 1).astype(np.float32)

    check(ctx, clump(nx), clump(ny), 100.0, 12, 30.0, False)


def test_lists_beyond_shared_memory(ctx):
    x = catalog.uniform(24, 20.0, seed=3)
    y = catalog.uniform(8200, 20.0, seed=4)
    for c in (x, y):
        c[:, :3] += 40.0
    gx, gy = ctx.grid(x, 100.0), ctx.grid(y, 100.0)
    for bins in (12, 33):
        np.testing.assert_array_equal(ctx.count_triplets(gx, gy, bins=bins, dmax=33.0),
                                      oracle.triplets_iso(x, y, box=100.0, bins=bins, dmax=33.0))


@pytest.mark.parametrize("dmax", [230.7, 700.3, 30000.7])
@pytest.mark.parametrize("bpc", [False, True])
def test_large_dmax(ctx, dmax, bpc):
    """bins / dmax is rounded down to 1e-6: the last bin's edge lies up to
    dmax * 1e-6 bins beyond dmax, inside and outside the edge windows."""
    box = 3.4 * dmax
    x = catalog.uniform(420, box, seed=11)
    y = catalog.uniform(400, box, seed=12)
    check(ctx, x, y, box, 13, dmax, bpc)


def test_many_stencil_rows(ctx):
    x = catalog.neyman_scott(700, 250.0, seed=21)
    y = catalog.uniform(500, 250.0, seed=22)
    check(ctx, x, y, 250.0, 30, 80.0, True, partitions=35)
    check(ctx, x, y, 250.0, 30, 80.0, False, partitions=50)
