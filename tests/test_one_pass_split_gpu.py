"""The one-pass smoothing's split of a level over the CTAs: boxes whose z
extent leaves a CTA part of one y-tile and part of the next, whose last tile
or CTA gets a short rest, and which need fewer CTAs than there are SMs, equal
the colour sweeps bit for bit, residual histories included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mx,minlevel", [((256, 64, 20), -1), ((256, 16, 4), -1), ((256, 200, 72), -2),
                                         ((256, 104, 200), -2)])
def test_one_pass_smoothing_across_tiles(pkg, ctx, mx, minlevel):
    out = {}
    for kind in (1, 3):
        h = pkg.Hierarchy(ctx, 3, 2, "ch", [5e-4, 0.02])
        h.build_uniform(list(mx), minlevel, [2] * 6, [0, 0, 0], [1, mx[1] / mx[0], mx[2] / mx[0]])
        h.commit()
        h.set_box_sweep(kind)
        h.seed_spinodal(0, 29, mean=0.1, amp=0.05)
        hist = [h.time_step(s == 0, 0, minlevel, tol=1e-12, maxvcycles=4, mode="mixed", strict=False)
                for s in range(2)]
        out[kind] = (hist, h.get(0, "q"))
        h.close()
    assert out[1][0] == out[3][0]
    assert np.array_equal(out[1][1], out[3][1])
