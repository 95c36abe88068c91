"""CPU: which blocks of the node-gate table hold the geometry of their images.
The corrections of the gated counts enumerate the others from the neighbours
through an image of anchors near two faces, so each must join both points
through images that involve two axes."""
from test_node_gates import _table


def test_blocks_without_the_geometry_of_their_images():
    t = _table("desi_b200/csrc/node_gates.cuh", "kGateBlocks[64]")
    by = _table("desi_b200/csrc/node_gates.cuh", "kGateByImage[64][2]")
    size = len(t) // 64
    irregular = set()
    for f3 in range(8):
        for f2 in range(8):
            b0, b1 = by[2 * (f2 | f3 << 3):][:2]
            ok = b0 >= 0 and b1 < 0
            if ok:
                B = t[size * b0:size * (b0 + 1)]
                pairs = set()
                ok = list(B[:4]) == [f2, f3, f2, f3]
                for k in range(3):
                    pair, n, *ax = B[4 + 5 * k:9 + 5 * k]
                    ax = [a for a in ax if a >= 0]
                    want = (f2, f2 ^ f3, f3)[pair]
                    ok = ok and n == len(ax) == bin(want).count("1") and sum(1 << a for a in set(ax)) == want
                    pairs.add(pair)
                ok = ok and pairs == {0, 1, 2}
            if not ok:
                irregular.add((f2, f3))
    assert irregular == {(3, 3), (5, 5), (6, 6), (7, 7), (1, 7), (2, 7), (3, 4), (7, 5)}
    assert all(f2 and f3 and bin(f2 | f3).count("1") >= 2 for f2, f3 in irregular)
