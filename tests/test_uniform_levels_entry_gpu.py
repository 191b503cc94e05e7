"""Uniform levels (kern_uni.cuh) against the oracle: rows beyond a wall under a
quasi-periodic offset, calls on a state whose ghosts the caller did not set,
and a V-cycle without smoothing."""
import numpy as np
import pytest

from tests.test_uniform_levels_gpu import BIO, CH2, CH3, GROWTH, PX, W

pytestmark = pytest.mark.gpu

# (problem, extents, minlevel, periodic or wall per dimension, qpo): a level
# or more above the cluster's 6144 cells, all of them in it, one row a CTA
QPO = {
    "2d-bio": (BIO, (48, 32), -3, (PX, W), [0.25, -0.5]),
    "2d-bio-above": (BIO, (128, 96), -4, (PX, W), [0.25, -0.5]),
    "2d-bio-thin": (BIO, (16, 64), -2, (PX, W), [0.25, 0.125]),
    "3d-walls": (CH3, (16, 12, 16), -2, (PX, W, W), [0.25, -0.5]),
    "3d-wall-z": (CH3, (16, 24, 12), -1, (PX, PX, W), [0.25, -0.5]),
    "3d-above": (CH3, (32, 24, 20), -2, (PX, W, W), [0.25, -0.5]),
    "3d-growth": (GROWTH, (16, 16, 12), -2, (PX, W, W), [0.25, -0.5, 0.75]),
}
STALE = {
    "2d-wall": (CH2, (40, 24), -3, (W, W), None),
    "2d-above": (CH2, (96, 80), -3, (W, PX), None),
    "2d-periodic": (CH2, (32, 48), -3, (PX, PX), None),
    "2d-bio": (BIO, (72, 40), -3, (W, W), None),
    "2d-bio-qpo": (BIO, (48, 32), -3, (PX, W), [0.25, -0.5]),
    "3d-wall": (CH3, (20, 12, 28), -2, (W, W, W), None),
    "3d-mixed": (CH3, (16, 12, 16), -2, (PX, W, PX), None),
    "3d-growth": (GROWTH, (24, 16, 12), -2, (W, W, W), None),
}


def build(mod, spec, ctx=None):
    (prob, prm, nv), n, mn, bc, qpo = spec
    nd = len(n)
    args = (nd, nv, prob, prm, qpo)
    h = mod.Hierarchy(ctx, *args) if ctx is not None else mod.OracleHierarchy(*args)
    faces = [b for b in bc for _ in range(2)] + [10] * (6 - 2 * nd)
    h.build_uniform(list(n) + [1] * (3 - nd), mn, faces, [0, 0, 0], [v / n[0] for v in n] + [1] * (3 - nd))
    h.commit()
    return h


def pair(pkg, ctx, oracle_mod, spec, seed):
    """the two hierarchies with the same random q, qold and f, ghosts included"""
    hs = build(pkg, spec, ctx), build(oracle_mod, spec)
    rng = np.random.default_rng(seed)
    for pid in range(0, -spec[2] + 1):
        for fld in ("q", "qold", "f"):
            a = rng.uniform(-1, 1, size=hs[0].field_size(pid, fld))
            for h in hs:
                h.put(pid, fld, a)
    return hs


def same_bits(g, o, spec, fields):
    for pid in range(0, -spec[2] + 1):
        for fld in fields:
            a, b = g.get(pid, fld), o.get(pid, fld)
            if a.size:
                assert np.array_equal(a, b), (pid, fld, int(np.sum(a != b)))


@pytest.mark.parametrize("case", list(QPO))
def test_offset_across_x_beside_a_wall(pkg, ctx, oracle_mod, case):
    g, o = pair(pkg, ctx, oracle_mod, QPO[case], 11)
    mn = QPO[case][2]
    for h in (g, o):
        h.set_ghost(0, 0)
        h.fill_down("q", 0, mn)
        h.fill_down("f", 0, mn)
        h.copy_q_to_qold(mn, 0)
        for _ in range(2):
            h.vcycle(0, mn, 2)
    same_bits(g, o, QPO[case], ("q", "qc", "f", "rf"))
    g.close()


@pytest.mark.parametrize("tail", [2048, 0])
@pytest.mark.parametrize("case", list(STALE))
def test_ghosts_the_caller_did_not_set(pkg, ctx, oracle_mod, case, tail):
    """LevelRelax and the V-cycle read the ghosts they find in their first
    colour sweep and SetGhost's from then on (afasroutines.f90:532-557)."""
    spec = STALE[case]
    mn = spec[2]
    for call in (lambda h: h.level_relax(0, 1), lambda h: h.level_relax(mn, 2), lambda h: h.vcycle(0, mn, 2),
                 lambda h: h.vcycle(-1, mn, 1),
                 lambda h: h.multigrid_iterations(0, mn, nsmooth=2, maxvcycles=2, tol=1e-300)):
        g, o = pair(pkg, ctx, oracle_mod, spec, 12)
        g.set_tail_cells(tail)
        call(g), call(o)
        same_bits(g, o, spec, ("q", "f"))
        g.close()


@pytest.mark.parametrize("tail", [2048, 0])
@pytest.mark.parametrize("case", list(STALE))
def test_vcycle_without_smoothing(pkg, ctx, oracle_mod, case, tail):
    spec = STALE[case]
    g, o = pair(pkg, ctx, oracle_mod, spec, 13)
    g.set_tail_cells(tail)
    for h in (g, o):
        h.set_ghost(0, 0)
        h.vcycle(0, spec[2], 0)
    same_bits(g, o, spec, ("q", "qc", "f", "rf"))
    g.close()
