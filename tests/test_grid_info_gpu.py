"""What a grid says of its cells: counts at sizes around a block and a warp of cells,
after the structure changed, and that asking again costs nothing."""
import time

import numpy as np
import pytest

from desi_b200 import catalog

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,P", [(1, 1), (1, 3), (40, 6), (300, 7), (5000, 16), (5000, 65), (20000, 161), (20000, 256)])
def test_counts(ctx, n, P):
    pts = catalog.neyman_scott(n, 100.0, seed=n, children=20)
    g = ctx.grid(pts, 100.0, partitions=P)
    want = np.count_nonzero(np.diff(g.download()[1]))
    assert g.info()["nonempty_cells"] == g.info()["nonempty_cells"] == want
    assert g.info()["partitions"] == P


def test_after_a_count_chose_other_cells(ctx):
    g = ctx.grid(catalog.uniform(4000, 100.0, seed=1), 100.0)
    seen = set()
    for dmax in (30.0, 9.0, 30.0, 3.0):
        ctx.count_pairs(g, bins=5, dmax=dmax)
        i = g.info()
        assert i["nonempty_cells"] == np.count_nonzero(np.diff(g.download()[1]))
        seen.add(i["partitions"])
    assert len(seen) > 1


def test_asking_again_is_free(ctx):
    """(the 64 MB cell table of 250 cells per side took 34 ms to fetch and walk)"""
    g = ctx.grid(catalog.uniform(4000, 100.0, seed=1), 100.0, partitions=250)
    g.info()
    t = []
    for _ in range(5):
        t0 = time.perf_counter()
        g.info()
        t.append(time.perf_counter() - t0)
    assert min(t) < 5e-3
