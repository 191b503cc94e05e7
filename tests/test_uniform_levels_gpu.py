"""Uniform levels (the single-patch levels <= 0): operations that write their
own ghost images, one launch each or as one cluster launch of the coarse
V-cycle.  The FP64 path has the oracle's bits in every field, ghosts
included, over boundary-condition mixes, ragged extents, extents of 2 and
quasi-periodic offsets; the correction cycle gives the same iterates whether
its coarse levels run in the cluster or one launch each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, PX = 10, 2
CH2, CH3 = ("ch", [1e-3, 0.02], 2), ("ch", [5e-4, 0.02], 2)
BIO, GROWTH = ("biogrowth", [0.1, 0.05, 1.5, 2.0, 0.5], 2), ("growth", [0.01, 0.025, 1.5, 2.0, 0.5, 1.0], 3)

# (problem, extents, minlevel, periodic or wall per dimension, qpo)
CASES = {
    "2d-periodic-tall": (CH2, (16, 96), -3, (PX, PX), None),        # uneven rows per CTA
    "2d-periodic-wide": (CH2, (200, 56), -2, (PX, PX), None),
    "2d-wall-odd-coarse": (CH2, (40, 24), -3, (W, W), None),         # coarsest 5 x 3
    "2d-x-periodic": (CH2, (48, 80), -3, (PX, W), None),
    "2d-y-periodic": (CH2, (36, 64), -2, (W, PX), None),
    "2d-qpo": (CH2, (32, 32), -4, (PX, W), [0.25, -0.5]),
    "2d-extent-2": (CH2, (4, 64), -1, (PX, PX), None),
    "2d-one-level": (CH2, (14, 10), 0, (PX, W), None),
    "2d-bio": (BIO, (72, 40), -3, (W, W), None),
    "2d-bio-periodic": (BIO, (64, 64), -5, (PX, PX), None),
    "3d-periodic": (CH3, (16, 24, 40), -2, (PX, PX, PX), None),
    "3d-wall": (CH3, (20, 12, 28), -2, (W, W, W), None),
    "3d-mixed": (CH3, (16, 12, 16), -2, (PX, W, PX), None),
    "3d-flat": (CH3, (32, 16, 4), -1, (W, PX, W), [0.5, 0.125]),
    "3d-growth": (GROWTH, (24, 16, 12), -2, (W, W, W), None),
}


def build(mod, case, ctx=None):
    (prob, prm, nv), n, mn, bc, qpo = CASES[case]
    nd = len(n)
    args = (nd, nv, prob, prm, qpo)
    h = mod.Hierarchy(ctx, *args) if ctx is not None else mod.OracleHierarchy(*args)
    faces = [b for b in bc for _ in range(2)] + [10] * (6 - 2 * nd)
    h.build_uniform(list(n) + [1] * (3 - nd), mn, faces, [0, 0, 0], [v / n[0] for v in n] + [1] * (3 - nd))
    h.commit()
    return h


def fill(hs, case, seed):
    _, n, mn, _, _ = CASES[case]
    rng = np.random.default_rng(seed)
    for pid in range(0, -mn + 1):
        for fld in ("q", "qold", "f"):
            a = rng.uniform(-1, 1, size=hs[0].field_size(pid, fld))
            for h in hs:
                h.put(pid, fld, a)


def same_bits(g, o, case, fields):
    for pid in range(0, -CASES[case][2] + 1):
        for fld in fields:
            a, b = g.get(pid, fld), o.get(pid, fld)
            if a.size:
                assert np.array_equal(a, b), (pid, fld, int(np.sum(a != b)))


@pytest.mark.parametrize("case", list(CASES))
def test_fp64_vcycle_has_the_oracles_bits(pkg, ctx, oracle_mod, case):
    g, o = build(pkg, case, ctx), build(oracle_mod, case)
    fill((g, o), case, 5)
    mn = CASES[case][2]
    for h in (g, o):
        h.set_ghost(0, 0)
        h.fill_down("q", 0, mn)
        h.fill_down("f", 0, mn)
        h.copy_q_to_qold(mn, 0)
    same_bits(g, o, case, ("q", "f"))
    for h in (g, o):
        h.vcycle(0, mn, 2)
    same_bits(g, o, case, ("q", "qc", "f", "rf"))
    g.set_tail_cells(0)  # every operation its own launch
    for h in (g, o):
        h.vcycle(0, mn, 1)
        h.level_relax(mn, 1)
    same_bits(g, o, case, ("q", "qc", "f", "rf"))
    g.close()


@pytest.mark.parametrize("case", ["2d-periodic-tall", "2d-wall-odd-coarse", "2d-bio", "3d-wall", "3d-growth"])
def test_fp64_step_leaves_every_level_as_the_oracle(pkg, ctx, oracle_mod, case):
    """FillDown of q and f below level 0 runs once after the last cycle."""
    g, o = build(pkg, case, ctx), build(oracle_mod, case)
    fill((g, o), case, 6)
    mn = CASES[case][2]
    for step in range(2):
        ng, _ = g.time_step(step == 0, 0, mn, tol=1e-9, maxvcycles=4)
        no, _ = o.time_step(step == 0, 0, mn, tol=1e-9, maxvcycles=4)
        assert ng == no
    same_bits(g, o, case, ("q", "qold", "f"))
    g.close()


@pytest.mark.parametrize("case", [c for c in CASES if not c.startswith("2d-bio")])
def test_mixed_cluster_equals_launches(pkg, ctx, case):
    """The two forms compute each cell alike; compiled apart, their FP32
    multiply-adds may round differently: 1e-9 of the solution's size, a
    hundredth of what the last cycle changes."""
    out = []
    for cells in (2048, 0):
        h = build(pkg, case, ctx)
        h.set_tail_cells(cells)
        n = CASES[case][1]
        rng = np.random.default_rng(8)
        h.put(0, "q", 0.1 * rng.uniform(-1, 1, size=h.field_size(0, "q")))
        n = [h.time_step(s == 0, 0, CASES[case][2], tol=1e-8, maxvcycles=8, mode="mixed")[0] for s in range(2)]
        out.append((n, h.get(0, "q")))
        h.close()
    assert out[0][0] == out[1][0]
    assert np.max(np.abs(out[0][1] - out[1][1])) <= 1e-9 * max(1.0, np.max(np.abs(out[1][1])))


# (extents, minlevel): rows dealt unevenly, one shared level, none, pairs of
# two cells a row, one level only, levels too large for the cluster above it
BOXES = [((16, 96), -3), ((200, 56), -2), ((4, 64), -1), ((2, 2), 0), ((20, 20), 0), ((34, 50), 0), ((128, 128), -6),
         ((256, 192), -5), ((16, 24, 40), -2), ((32, 32, 32), -4), ((4, 4, 64), -1), ((6, 10, 2), 0), ((64, 48, 32), -3)]


@pytest.mark.parametrize("n,mn", BOXES)
def test_box_solve_reaches_the_fp64_solution(pkg, ctx, n, mn):
    """Mixed steps on periodic boxes, converged tightly, against the FP64
    path: the residual 1e-11 bounds the difference by about 1e-11 over the
    operator's smallest eigenvalue (one), 1e-9 is a hundred times that."""
    nd = len(n)
    q = {}
    for mode in ("fp64", "mixed"):
        h = pkg.Hierarchy(ctx, nd, 2, "ch", [1e-5, 0.05])
        h.build_uniform(list(n) + [1] * (3 - nd), mn, [2] * (2 * nd) + [10] * (6 - 2 * nd), [0, 0, 0],
                        [v / n[0] for v in n] + [1] * (3 - nd))
        h.commit()
        h.seed_spinodal(0, 3)
        for s in range(3):
            _, res = h.time_step(s == 0, 0, mn, tol=1e-11, maxvcycles=40, mode=mode)
            assert res[-1] < 1e-11
        q[mode] = h.get(0, "q")
        h.close()
    assert np.max(np.abs(q["mixed"] - q["fp64"])) <= 1e-9


@pytest.mark.parametrize("errortype", [1, 2])
@pytest.mark.parametrize("n,mn", BOXES)
def test_box_solve_in_one_launch_equals_the_host_loop(pkg, ctx, n, mn, errortype):
    """A V-cycle limit above 64 takes the loop of separate launches; up to 64
    a box that fits is one launch.  Both compute each cell alike (1e-9 of the
    solution's size, as above), ghosts included; their norms add in another
    order, in single precision over a thread's and a warp's cells."""
    nd = len(n)
    out = []
    for most in (64, 65):
        h = pkg.Hierarchy(ctx, nd, 2, "ch", [1e-5, 0.05])
        h.build_uniform(list(n) + [1] * (3 - nd), mn, [2] * (2 * nd) + [10] * (6 - 2 * nd), [0, 0, 0],
                        [v / n[0] for v in n] + [1] * (3 - nd))
        h.commit()
        h.seed_spinodal(0, 3)
        steps = [h.time_step(s == 0, 0, mn, tol=1e-9, maxvcycles=most, errortype=errortype, mode="mixed")
                 for s in range(3)]
        out.append((steps, [h.get(p, "q") for p in range(-mn + 1)]))
        h.close()
    for (na, ra), (nb, rb) in zip(out[0][0], out[1][0]):
        assert na == nb
        assert np.allclose(ra, rb, rtol=1e-4, atol=0)
    for a, b in zip(out[0][1], out[1][1]):
        assert np.max(np.abs(a - b)) <= 1e-9 * max(1.0, np.max(np.abs(b)))
