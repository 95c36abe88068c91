"""Captured batches are told apart by every bit of dmax: two calls on the same
grids whose dmax differ in the last bit only, with pairs between the two, each
return their own histogram."""
import numpy as np
import pytest

from desi_b200 import catalog

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ani", [False, True])
def test_neighbouring_dmax(ctx, ani):
    box, bins = 300.0, 15
    below = np.float32(97.5)
    above = np.nextafter(below, np.float32(200.0))
    # pairs along x at a distance of exactly 97.5: out of range of the first, in
    # range of the second (a little off the axis, so that no component is zero)
    D, R = catalog.uniform(300, box, seed=1), catalog.uniform(310, box, seed=2)
    D[:40, 0], R[:40, 0] = 16.0, 16.0 + below
    D[:40, 1:3] = np.arange(40, dtype=np.float32)[:, None] * 7.0 + 4.0
    R[:40, 1:3] = D[:40, 1:3]
    gd, gr = ctx.grid(D, box), ctx.grid(R, box)
    flags = 0
    if ani:  # the rule without the exclusion of zero components
        from desi_b200 import api
        flags = api.PCF_RULE_CUSTOM
    kw = dict(bins=bins, ani=ani, flags=flags)
    plain = [ctx.batch_pairs(gd, [gr], dmax=float(d), **kw) for d in (below, above)]
    assert plain[1][2].sum() >= plain[0][2].sum() + 40
    for _ in range(2):  # captured, then replayed
        for d, want in zip((below, above), plain):
            got = ctx.batch_pairs(gd, [gr], dmax=float(d), graph=True, **kw)
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g, w)
