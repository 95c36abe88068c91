"""The fine pair histograms of the closed-form 3iso stop on an abort request: the
call (without a counted DDD, so theirs is the only queue) returns PCF_ERR_TIMEOUT,
and the context counts as before once the request is cleared."""
import numpy as np
import pytest

from desi_b200 import api, catalog

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weights", ["unit", "uniform"])
@pytest.mark.parametrize("n", [40, 3000])
def test_fine_counts_poll_the_abort_word(n, weights):
    D = catalog.neyman_scott(n, 250.0, seed=5, weights=weights)
    kw = dict(bins=8, dmax=60.0, with_ddd=False)
    c = api.Context(0)
    try:
        g = c.grid(D, 250.0)
        before = c.analytic_3iso(g, **kw)[1:]
        c.set_option(api.PCF_OPT_ABORT_HOST_CHECK, 0)
        c.abort(True)
        with pytest.raises(api.PcfError) as e:
            c.analytic_3iso(g, **kw)
        assert e.value.status == api.PCF_ERR_TIMEOUT
        c.abort(False)
        c.set_option(api.PCF_OPT_ABORT_HOST_CHECK, 1)
        for a, b in zip(c.analytic_3iso(g, **kw)[1:], before):
            np.testing.assert_allclose(a, b, rtol=1e-12, atol=0)
        c.synchronize()
    finally:
        c.close()
