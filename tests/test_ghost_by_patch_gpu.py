"""Ghost programs compiled a patch at a time, and the general analysis that
remains for a level whose patches overlap: SetGhost of every pass against the
oracle's sequential writers, bit for bit, over adjacent, touching-by-corner,
edge and overlapping patches, periodic images and walls, one ghost layer and
two."""
import numpy as np
import pytest

from hierarchies import Spec

pytestmark = pytest.mark.gpu

P2, W2 = [2] * 4 + [10] * 2, [10] * 6
P3, M3 = [2] * 6, [2, 2, 10, 10, 2, 2]
# (ndims, boundary codes, children of the root as (lo, hi) in its cells)
CASES = {
    "2d-adjacent": (2, P2, [((3, 3), (6, 6)), ((7, 3), (10, 8)), ((5, 9), (8, 12))]),
    "2d-edges": (2, P2, [((1, 1), (4, 4)), ((13, 13), (16, 16)), ((13, 1), (16, 6)), ((1, 9), (2, 12))]),
    "2d-walls": (2, W2, [((1, 1), (4, 4)), ((5, 1), (8, 2)), ((9, 9), (16, 16))]),
    "2d-overlap": (2, P2, [((3, 3), (8, 8)), ((6, 6), (11, 11)), ((1, 1), (2, 16))]),
    "2d-overlap-image": (2, P2, [((1, 1), (16, 4)), ((9, 9), (12, 12)), ((11, 10), (16, 12))]),
    "3d-adjacent": (3, P3, [((1, 1, 1), (4, 4, 4)), ((5, 1, 1), (8, 4, 4)), ((5, 5, 5), (8, 8, 8))]),
    "3d-mixed": (3, M3, [((1, 1, 3), (2, 8, 6)), ((7, 1, 1), (8, 2, 8)), ((3, 3, 3), (4, 4, 4))]),
    "3d-overlap": (3, P3, [((2, 2, 2), (5, 5, 5)), ((4, 4, 4), (7, 7, 7)), ((7, 1, 1), (8, 8, 3))]),
}


@pytest.mark.parametrize("mbc", [1, 2])
@pytest.mark.parametrize("case", list(CASES))
def test_set_ghost_has_the_oracles_bits(pkg, ctx, oracle_mod, case, mbc):
    nd, bc, kids = CASES[case]
    s = Spec(nd)
    s.root_and_below(16 if nd == 2 else 8, -1, bc)
    for x, (lo, hi) in enumerate(kids):
        s.child(0, 10 + x, lo, hi)
    hs = [pkg.Hierarchy(ctx, nd, 2, "ch", [1e-3, 0.02], mbc=mbc),
          oracle_mod.OracleHierarchy(nd, 2, "ch", [1e-3, 0.02], mbc=mbc)]
    for h in hs:
        s.apply(h)
    rng = np.random.default_rng(4)
    ids = [p["id"] for p in s.patches]
    for ipass in (0, 1, 2):
        for i in ids:
            a = rng.uniform(-1, 1, size=hs[0].field_size(i, "q"))
            for h in hs:
                h.put(i, "q", a)
        for h in hs:
            h.set_ghost(1, ipass)
        for i in ids:
            assert np.array_equal(hs[0].get(i, "q"), hs[1].get(i, "q")), (ipass, i)
    hs[0].close()
