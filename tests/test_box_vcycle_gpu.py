"""One V-cycle of the periodic box's correction form, cell by cell, against
one V-cycle of the FP64 path from the same state, which has the oracle's bits.
The two are the same algebra: they differ by the FP32 rounding of the
correction.  That covers the whole solve in one cluster launch, the cluster's
V-cycle below levels of separate launches, and the one-launch partition's
forms (rows dealt unevenly, one row a CTA, levels held by every second CTA, by
CTA 0 alone)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOXES = [((32, 32), -4), ((128, 128), -6), ((96, 64), -4), ((40, 48), -2), ((64, 22), 0), ((256, 16), -3),
         ((16, 256), -3), ((512, 384), -6), ((32, 32, 32), -4), ((24, 16, 24), -2), ((64, 32, 16), -3),
         ((8, 48, 40), -2), ((64, 64, 64), -5), ((96, 80, 64), -3)]


@pytest.mark.parametrize("n,mn", BOXES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_one_cycle_agrees_with_fp64(pkg, ctx, n, mn):
    """The limit: 2^-24 an operation, a thousand of them in a row (a cell's
    chain through the levels of 12 or so half-sweeps of 20 operations each,
    down and up, at most seven levels), errors that do not cancel: 6e-5 of the
    largest change.  A halo or a row taken from the wrong place is off by the
    order of the change itself."""
    nd = len(n)
    out = []
    for mode in ("fp64", "mixed"):
        h = pkg.Hierarchy(ctx, nd, 2, "ch", [1e-3, 0.02])
        h.build_uniform(list(n) + [1] * (3 - nd), mn, [2] * (2 * nd) + [10] * (6 - 2 * nd), [0, 0, 0],
                        [v / n[0] for v in n] + [1] * (3 - nd))
        h.commit()
        h.seed_spinodal(0, 5, mean=0.1, amp=0.3)
        h.set_ghost(0, 0)
        before = h.get(0, "q")
        h.time_step(True, 0, mn, tol=1e-30, maxvcycles=1, mode=mode)
        out.append(h.get(0, "q"))
        h.close()
    change = np.max(np.abs(out[0] - before))
    off = np.max(np.abs(out[1] - out[0]))
    print(n, change, off / change)
    assert off <= 6e-5 * change
