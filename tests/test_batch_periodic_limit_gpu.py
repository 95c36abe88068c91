"""A periodic batch refuses what a single periodic call refuses: a dmax so close
to half the box that no cell size of the library keeps the stencil from wrapping
onto itself.  Below that it counts every pair, those across the box among them."""
import numpy as np
import pytest

import oracle
from desi_b200 import api, catalog

pytestmark = pytest.mark.gpu
PCF_ERR_UNSUPPORTED = -4


@pytest.mark.parametrize("ani", [False, True, "both"])
@pytest.mark.parametrize("dmax", [40.0, 48.5, 49.0, 49.3, 49.6, 49.9, 49.99])
def test_batch_as_single_calls(ctx, dmax, ani):
    box, bins = 100.0, 9
    D, R = catalog.uniform(500, box, seed=3), catalog.uniform(450, box, seed=4)
    # neighbours in two cells around the middle, and partners just inside dmax of
    # one of them through either face
    D[:2, :3] = [[30.0, 30.0, 49.7], [30.0, 30.0, 50.3]]
    R[:2, :3] = [[30.0, 30.0, 0.1], [30.0, 30.0, 99.9]]
    gd, gr = ctx.grid(D, box), ctx.grid(R, box)
    kw = dict(bins=bins, dmax=dmax, ani=ani, bpc=True)
    try:
        single = ctx.count_pairs(gd, gr, **kw)
    except api.PcfError as e:
        assert e.status == PCF_ERR_UNSUPPORTED
        single = None
    if single is None:
        for graph in (False, True):
            with pytest.raises(api.PcfError) as e:
                ctx.batch_pairs(gd, [gr], graph=graph, **kw)
            assert e.value.status == PCF_ERR_UNSUPPORTED
        return
    dr = ctx.batch_pairs(gd, [gr], **kw)[2]
    if ani == "both":
        dr, kinds = (dr[0][0], dr[1][0]), (False, True)
    else:
        dr, single, kinds = (dr[0],), (single,), (ani,)
    for got, one, k in zip(dr, single, kinds):
        np.testing.assert_array_equal(got, one)
        np.testing.assert_array_equal(got, oracle.pairs(D, R, box=box, bins=bins, dmax=dmax, ani=k, bpc=True))


def test_some_are_refused_and_some_are_not(ctx):
    g = ctx.grid(catalog.uniform(500, 100.0, seed=3), 100.0)
    ctx.batch_pairs(g, [g], bins=9, dmax=48.5, bpc=True)
    with pytest.raises(api.PcfError):
        ctx.batch_pairs(g, [g], bins=9, dmax=49.9, bpc=True)
