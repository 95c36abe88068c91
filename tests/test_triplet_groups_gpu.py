"""Triplet counts of a dense clump in a large box, whose lists are far longer than the
catalogs' mean density says: the histograms, and that few anchors do not take three
times the scratch."""
import numpy as np
import pytest

import oracle
from desi_b200 import _lib, api, catalog

pytestmark = pytest.mark.gpu


def _clump(n, box, seed, weights="unit"):
    p = catalog.uniform(n, box, seed=seed, weights=weights)
    g = np.random.default_rng(seed)
    p[:, :3] = box / 2 + 12.0 * np.clip(g.standard_normal((n, 3)), -3.0, 3.0)
    return p


@pytest.mark.parametrize("weights", ["unit", "uniform"])
@pytest.mark.parametrize("nx,ny", [(60, 8192), (60, 8193), (150, 12000), (2700, 9000)])
def test_values(ctx, nx, ny, weights):
    box, bins, dmax = 1000.0, 6, (12.0 if nx < 1000 else 2.0)
    X, Y = _clump(nx, box, 1, weights), _clump(ny, box, 2, weights)
    gx, gy = ctx.grid(X, box), ctx.grid(Y, box)
    for y, Q in ((None, None), (gy, Y)):
        got = ctx.count_triplets(gx, y, bins=bins, dmax=dmax)
        want = oracle.triplets_iso(X, Q, box=box, bins=bins, dmax=dmax)
        np.testing.assert_allclose(got, want, rtol=0 if weights == "unit" else 1e-12, atol=0)


def test_scratch_of_few_anchors():
    """800 anchors against a clump of 60000 points: one list of each kind per SM (284 MB;
    three of each took 853)."""
    c = api.Context(0)
    try:
        gx, gy = c.grid(_clump(800, 1000.0, 1), 1000.0), c.grid(_clump(60000, 1000.0, 2), 1000.0)
        c.count_triplets(gx, None, bins=20, dmax=25.0)
        before = _lib.alloc_counters()["device_bytes"]
        c.count_triplets(gx, gy, bins=20, dmax=25.0)
        assert _lib.alloc_counters()["device_bytes"] - before < 500e6
    finally:
        c.close()
