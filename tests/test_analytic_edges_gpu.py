"""The analytic 3iso path at sub-grids and catalogs where its fine histograms and
its interval ends can go wrong: a sub-grid finer than a block, or of a few cells,
one bin, dmax near half the box, a few points, and weights."""
import numpy as np
import pytest

import oracle
from desi_b200 import catalog
from desi_b200._lib import PcfError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box,bins,dmax,ptt,bn_ref", [
    (2, 100.0, 1, 49.0, 100, 5), (33, 100.0, 3, 45.0, 1, 1), (700, 250.0, 3, 60.1, 3, 41), (400, 64.0, 5, 16.0, 10, 16)])
@pytest.mark.parametrize("weights", ["unit", "uniform"])
def test_sub_grids(ctx, n, box, bins, dmax, ptt, bn_ref, weights):
    D = catalog.neyman_scott(n, box, seed=n, children=max(1, n // 5), weights=weights)
    _, ddr, rrr = ctx.analytic_3iso(ctx.grid(D, box), bins=bins, dmax=dmax, ptt=ptt, bn_ref=bn_ref, with_ddd=False)
    oddr, orrr, _, _ = oracle.analytic_3iso(D, box=box, bins=bins, dmax=dmax, ptt=ptt, bn_ref=bn_ref)
    # sums of bn_ref^3 terms in another order (the existing tests' bounds)
    np.testing.assert_allclose(rrr, orrr, rtol=1e-10, atol=1e-12 * np.abs(orrr).max())
    np.testing.assert_allclose(ddr, oddr, rtol=1e-10, atol=1e-12 * np.abs(oddr).max())


def test_one_point(ctx):
    """No pairs: DD / RR - 1 is -1 everywhere, and DDR vanishes up to rounding."""
    D = catalog.uniform(1, 100.0, seed=1)
    ddd, ddr, rrr = ctx.analytic_3iso(ctx.grid(D, 100.0), bins=2, dmax=30.0, ptt=4, bn_ref=3)
    assert not ddd.any() and rrr.any()
    assert np.abs(ddr).max() <= 1e-12 * rrr.max()


def test_no_periodic_stencil(ctx):
    with pytest.raises(PcfError, match="box/2"):
        ctx.analytic_3iso(ctx.grid(catalog.uniform(500, 100.0, seed=2), 100.0), bins=4, dmax=49.9, with_ddd=False)


def test_a_sub_grid_finer_than_a_block(ctx):
    box, bins, dmax, bn_ref = 100.0, 3, 30.0, 300
    D = catalog.uniform(900, box, seed=3)
    _, ddr, rrr = ctx.analytic_3iso(ctx.grid(D, box), bins=bins, dmax=dmax, ptt=5, bn_ref=bn_ref, with_ddd=False)
    _, ffr, alpha = oracle.analytic_ff(D, box=box, bins=bins, dmax=dmax, ptt=5, bn_ref=bn_ref)
    for i, j, k in ((0, 0, 1), (1, 2, 2), (0, 1, 1)):
        v, r, d = oracle.analytic_bin(i, j, k, bins=bins, dmax=dmax, bn_ref=bn_ref, alpha_ref=alpha, ff_ref=ffr)
        if 0 < v < 8:
            np.testing.assert_allclose([rrr[i, j, k], ddr[i, j, k]], [r, d], rtol=1e-10)
