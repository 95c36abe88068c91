"""A batch of many small catalogs by the branch-free pair kernel: its histograms, and
that exact weights cost no more than signed ones, which the general kernel counts."""
import time

import numpy as np
import pytest

import oracle
from desi_b200 import catalog

pytestmark = pytest.mark.gpu


def _catalogs(weights, nr=100):
    D = catalog.neyman_scott(1000, 500.0, seed=18, weights="unit" if weights == "unit" else "uniform")
    Rs = [catalog.uniform(250 + 7 * i, 500.0, seed=20 + i, weights="unit" if weights == "unit" else "uniform")
          for i in range(nr)]
    if weights == "signed":
        for p in [D] + Rs:
            p[::2, 3] *= -1.0
    return D, Rs


@pytest.mark.parametrize("ani", [False, True])
@pytest.mark.parametrize("weights", ["unit", "uniform"])
@pytest.mark.parametrize("graph", [False, True])
def test_values(ctx, weights, ani, graph):
    D, Rs = _catalogs(weights)
    gd, gr = ctx.grid(D, 500.0), [ctx.grid(R, 500.0) for R in Rs]
    for _ in range(2):  # (captured, then replayed)
        dd, rr, dr = ctx.batch_pairs(gd, gr, bins=25, dmax=50.0, ani=ani, bpc=True, graph=graph)
        kw = dict(box=500.0, bins=25, dmax=50.0, ani=ani, bpc=True)
        tol = dict(rtol=0 if weights == "unit" else 1e-12, atol=0)
        np.testing.assert_allclose(dd, oracle.pairs(D, None, **kw), **tol)
        for i in (0, 1, 2, 31, 62, 98, 99):
            np.testing.assert_allclose(rr[i], oracle.pairs(Rs[i], None, **kw), **tol)
            np.testing.assert_allclose(dr[i], oracle.pairs(D, Rs[i], **kw), **tol)


def test_exact_weights_cost_no_more_than_signed(ctx):
    """(with one job at a time per CTA, 1.4 to 1.5 times as much)"""
    t = {}
    calls = {}
    for w in ("uniform", "signed"):
        D, Rs = _catalogs(w)
        gd, gr = ctx.grid(D, 500.0), [ctx.grid(R, 500.0) for R in Rs]
        calls[w] = lambda gd=gd, gr=gr: ctx.batch_pairs(gd, gr, bins=25, dmax=50.0, graph=True)
        t[w] = []
    for k in range(12):
        for w, f in calls.items():
            t0 = time.perf_counter()
            f()
            t[w].append(time.perf_counter() - t0)
    assert min(t["uniform"]) <= 1.2 * min(t["signed"]), (min(t["uniform"]), min(t["signed"]))
