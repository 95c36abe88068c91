"""Weighted 3-point counts in three integer limbs: weights whose sums FP64 holds
exactly (then every bin is the oracle's), full mantissas (carries between all
limbs), weights of 0, a range of weights that has no exact integers or whose
products leave no room, bin counts around the shared histogram's limit, budgets
that flush it after every few anchors, lists that spill, and batches."""
import numpy as np
import pytest

import oracle
from desi_b200 import catalog
from desi_b200._lib import PCF_OPT_TRIP_FLUSH_BUDGET

pytestmark = pytest.mark.gpu


def weights(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "eighths":
        return rng.integers(1, 17, n) / 8.0
    if kind == "zeros":
        return rng.integers(0, 3, n) / 4.0
    if kind == "mantissa":
        return np.float32(1.0) + rng.random(n).astype(np.float32)
    if kind == "binades":  # q up to 2^32: no room for a product
        return rng.random(n).astype(np.float32) * np.exp2(rng.integers(0, 7, n)) + np.float32(0.5)
    return rng.random(n).astype(np.float32) * 10.0 ** rng.integers(-9, 9, n) * rng.choice([-1.0, 1.0], n)


def cat(points, kind, seed):
    p = points.copy()
    p[:, 3] = weights(kind, len(p), seed).astype(np.float32)
    return p


def check(ctx, D, R, bins, dmax, bpc, exact, box=100.0):
    gd, gr = ctx.grid(D, box), ctx.grid(R, box)
    for x, y, X, Y in ((gd, None, D, None), (gr, None, R, None), (gd, gr, D, R), (gr, gd, R, D)):
        got = ctx.count_triplets(x, y, bins=bins, dmax=dmax, bpc=bpc)
        want = oracle.triplets_iso(X, Y, box=box, bins=bins, dmax=dmax, bpc=bpc)
        if exact:
            np.testing.assert_array_equal(got, want)
        else:  # at most 1e5 terms a bin, each sum within terms * 2^-53
            np.testing.assert_allclose(got, want, rtol=2e-11, atol=2e-11 * np.abs(want).max())
    return gd, gr


@pytest.mark.parametrize("kind", ["eighths", "zeros", "mantissa", "binades", "signs"])
@pytest.mark.parametrize("bpc", [False, True])
@pytest.mark.parametrize("n,bins", [(2, 5), (3, 1), (40, 7), (230, 20)])
def test_weights(ctx, kind, bpc, n, bins):
    D = cat(catalog.neyman_scott(n, 100.0, seed=n, children=max(2, n // 4)), kind, 1)
    R = cat(catalog.uniform(n + 9, 100.0, seed=n + 1), kind, 2)
    check(ctx, D, R, bins, 33.0, bpc, kind in ("eighths", "zeros"))


@pytest.mark.parametrize("bins", [2, 29, 30, 31, 33])
def test_bin_counts(ctx, bins):
    D = cat(catalog.uniform(250, 100.0, seed=3), "eighths", 3)
    R = cat(catalog.uniform(200, 100.0, seed=4), "eighths", 4)
    check(ctx, D, R, bins, 40.0, True, True)


@pytest.mark.parametrize("budget", [1, 3000, 100000])
def test_flushes(ctx, budget):
    D = cat(catalog.neyman_scott(400, 100.0, seed=5), "mantissa", 5)
    R = cat(catalog.uniform(300, 100.0, seed=6), "eighths", 6)
    try:
        ctx.set_option(PCF_OPT_TRIP_FLUSH_BUDGET, budget)
        check(ctx, D, R, 12, 30.0, False, False)
    finally:
        ctx.set_option(PCF_OPT_TRIP_FLUSH_BUDGET, 1 << 31)


def test_batch_equals_single_counts(ctx):
    D = cat(catalog.neyman_scott(700, 100.0, seed=7), "eighths", 7)
    Rs = [cat(catalog.uniform(500 + 100 * k, 100.0, seed=8 + k), "eighths", 8 + k) for k in range(3)]
    gd, gr = ctx.grid(D, 100.0), [ctx.grid(r, 100.0) for r in Rs]
    kw = dict(bins=15, dmax=30.0, bpc=True)
    ddd, rrr, ddr, drr = ctx.batch_triplets(gd, gr, **kw)
    np.testing.assert_array_equal(ddd, ctx.count_triplets(gd, **kw))
    for k, g in enumerate(gr):
        np.testing.assert_array_equal(rrr[k], ctx.count_triplets(g, **kw))
        np.testing.assert_array_equal(ddr[k], ctx.count_triplets(gd, g, **kw))
        np.testing.assert_array_equal(drr[k], ctx.count_triplets(g, gd, **kw))


def test_lists_that_spill(ctx):
    """4000 points of one clump: lists past the shared room, against the same
    points with unit weights (2^-3 per triangle)."""
    rng = np.random.default_rng(10)
    p = np.ones((4000, 4), np.float32)
    p[:, :3] = 50.0 + rng.normal(0, 6.0, (4000, 3))
    h = p.copy()
    h[:, 3] = 0.5
    kw = dict(bins=30, dmax=40.0)
    a, b = ctx.grid(p, 100.0), ctx.grid(h, 100.0)
    np.testing.assert_array_equal(ctx.count_triplets(a, **kw), 8.0 * ctx.count_triplets(b, **kw))
    np.testing.assert_array_equal(ctx.count_triplets(a, a, **kw), 8.0 * ctx.count_triplets(b, b, **kw))
