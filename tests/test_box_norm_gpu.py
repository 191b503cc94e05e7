"""The width of the sums in the one-launch box solve's residual norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT, EPS = 1e-3, 0.02


def afas_norm(h, n, nv=2):
    """ErrorAFAS of Cahn-Hilliard in FP64 from q and qold (afasroutines.f90:113-233)"""
    nd = len(n)
    inner = (slice(1, -1),) * nd

    def lap(a):
        s = -2.0 * nd * a[inner]
        for d in range(nd):
            for o in (0, 2):
                s = s + a[tuple(slice(o, a.shape[d] - 2 + o) if x == d else slice(1, -1) for x in range(nd))]
        return s
    q = h.get(0, "q").reshape([v + 2 for v in n] + [nv], order="F")
    old = h.get(0, "qold").reshape([v + 2 for v in n] + [nv], order="F")
    phi, mu, f = q[..., 0], q[..., 1], old[..., 0][inner]
    h2 = (1.0 / n[0]) ** 2
    r0 = f - (phi[inner] - DT / h2 * lap(mu))
    r1 = -f - (mu[inner] - phi[inner] ** 3 + EPS**2 / h2 * lap(phi))
    return float(np.sqrt((np.sum(r0 * r0) + np.sum(r1 * r1)) / (2.0 * f.size)))


@pytest.mark.parametrize("n,mn", [((128, 128), -6), ((32, 32, 32), -4)])
def test_single_precision_sums_stay_within_a_warp(pkg, ctx, n, mn):
    """The norm adds squares of FP32 residuals, in FP32 over a warp's 64 (128)
    cells and in FP64 from there.  Rounding errors of such sums are random:
    simulated over both schedules with normal residuals, 1.2e-9 of the norm
    (rms); carried in FP32 to a CTA's 1024 (2048) cells, 4.5e-9.  The limit is
    their geometric mean."""
    nd = len(n)
    off = []
    h = pkg.Hierarchy(ctx, nd, 2, "ch", [DT, EPS])
    h.build_uniform(list(n) + [1] * (3 - nd), mn, [2] * (2 * nd) + [10] * (6 - 2 * nd), [0, 0, 0],
                    [v / n[0] for v in n] + [1] * (3 - nd))
    h.commit()
    for seed in range(96):
        h.seed_spinodal(0, seed + 1, mean=0.1, amp=0.3)
        _, res = h.time_step(True, 0, mn, tol=1e-30, maxvcycles=1, mode="mixed")
        off.append(res[-1] / afas_norm(h, n) - 1.0)
    h.close()
    rms = float(np.sqrt(np.mean(np.square(off))))
    print(n, rms)
    assert rms < 2.3e-9
