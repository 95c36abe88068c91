"""Separations within a few float32 roundings of a bin edge or of dmax: the
FP32 fast path must hand every one of them to the FP64 rule, directly and
through periodic images, for pairs and for the third side of a triangle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def edge_catalogs(box, bins, dmax, n, seed):
    """n points and n partners, partner i at a distance within 4 ulp of a bin
    edge (dmax among them), along an axis or a random direction, wrapped into
    the box; half of the points lie within dmax of a face."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.0, box, (n, 3))
    near = rng.random((n, 3)) < 0.5
    a[near] = np.where(rng.random(near.sum()) < 0.5, 1.0, -1.0) * rng.uniform(0.0, dmax, near.sum())
    a = np.mod(a, box).astype(np.float32)
    a[a >= np.float32(box)] = 0.0
    d = rng.normal(size=(n, 3))
    axis = rng.random(n) < 0.5
    d[axis] = np.eye(3)[rng.integers(0, 3, axis.sum())]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = rng.integers(1, bins + 1, n) * (dmax / bins) * (1.0 + rng.integers(-4, 5, n) * 2.0 ** -23)
    b = np.mod(a.astype(np.float64) + d * r[:, None], box).astype(np.float32)
    b[b >= np.float32(box)] = 0.0
    one = np.ones((n, 1), np.float32)
    return np.concatenate([a, one], 1), np.concatenate([b, one], 1)


@pytest.mark.parametrize("bpc", [False, True])
@pytest.mark.parametrize("box,bins,dmax", [(250.0, 30, 80.0), (1000.0, 41, 119.7), (2000.0, 20, 20.0), (97.0, 200, 31.3)])
def test_pairs_at_bin_edges(ctx, box, bins, dmax, bpc):
    a, b = edge_catalogs(box, bins, dmax, 1500, 5)
    ga, gb = ctx.grid(a, box), ctx.grid(b, box)
    both = np.concatenate([a, b])
    g2 = ctx.grid(both, box)
    for ani in (False, True):
        np.testing.assert_array_equal(
            ctx.count_pairs(ga, gb, bins=bins, dmax=dmax, ani=ani, bpc=bpc),
            oracle.pairs(a, b, box=box, bins=bins, dmax=dmax, ani=ani, bpc=bpc))
        np.testing.assert_array_equal(
            ctx.count_pairs(g2, None, bins=bins, dmax=dmax, ani=ani, bpc=bpc),
            oracle.pairs(both, None, box=box, bins=bins, dmax=dmax, ani=ani, bpc=bpc))


@pytest.mark.parametrize("bpc", [False, True])
@pytest.mark.parametrize("box,bins,dmax", [(250.0, 30, 80.0), (400.0, 13, 97.3)])
def test_triangles_at_bin_edges(ctx, box, bins, dmax, bpc):
    a, b = edge_catalogs(box, bins, dmax, 400, 6)
    ga, gb = ctx.grid(a, box), ctx.grid(b, box)
    g2 = ctx.grid(np.concatenate([a, b]), box)
    np.testing.assert_array_equal(
        ctx.count_triplets(g2, None, bins=bins, dmax=dmax, bpc=bpc),
        oracle.triplets_iso(np.concatenate([a, b]), None, box=box, bins=bins, dmax=dmax, bpc=bpc))
    np.testing.assert_array_equal(
        ctx.count_triplets(ga, gb, bins=bins, dmax=dmax, bpc=bpc),
        oracle.triplets_iso(a, b, box=box, bins=bins, dmax=dmax, bpc=bpc))
