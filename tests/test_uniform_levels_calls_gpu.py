"""FP64 calls on uniform levels in random order, on states and hierarchies of
random shape, against the oracle: every field of every level has its bits
after every call."""
import random

import numpy as np
import pytest

from tests.test_uniform_levels_gpu import BIO, CH2, CH3, GROWTH, PX, W

pytestmark = pytest.mark.gpu


def pair(pkg, ctx, oracle_mod, prob, n, mn, bc, qpo, seed):
    """the two hierarchies with the same random q, qold and f, ghosts included"""
    (name, prm, nv), nd = prob, len(n)
    hs = pkg.Hierarchy(ctx, nd, nv, name, prm, qpo), oracle_mod.OracleHierarchy(nd, nv, name, prm, qpo)
    rng = np.random.default_rng(seed)
    for h in hs:
        h.build_uniform(list(n) + [1] * (3 - nd), mn, [b for b in bc for _ in range(2)] + [10] * (6 - 2 * nd),
                        [0, 0, 0], [v / n[0] for v in n] + [1] * (3 - nd))
        h.commit()
    for pid in range(0, -mn + 1):
        for fld in ("q", "qold", "f"):
            a = rng.uniform(-1, 1, size=hs[0].field_size(pid, fld))
            for h in hs:
                h.put(pid, fld, a)
    return hs


def differences(g, o, mn):
    return [(pid, fld) for pid in range(0, -mn + 1) for fld in ("q", "qold", "qc", "f", "rf")
            if g.field_size(pid, fld) and not np.array_equal(g.get(pid, fld), o.get(pid, fld), equal_nan=True)]


@pytest.mark.parametrize("tail", [2048, 0])
@pytest.mark.parametrize("prob,n,mn,bc", [(CH2, (34, 122), 0, (W, PX)), (BIO, (64, 32), -4, (W, PX)),
                                          (CH3, (24, 24, 32), -3, (W, W, PX)), (GROWTH, (16, 8, 16), -2, (PX, PX, W))])
def test_a_vcycle_of_one_level_without_smoothing_changes_nothing(pkg, ctx, oracle_mod, prob, n, mn, bc, tail):
    g, o = pair(pkg, ctx, oracle_mod, prob, n, mn, bc, None, 3)
    g.set_tail_cells(tail)
    for level in (mn, 0):
        g.vcycle(level, level, 0), o.vcycle(level, level, 0)
        assert differences(g, o, mn) == []
    g.close()


@pytest.mark.parametrize("first", range(0, 160, 20))
def test_calls_in_random_order(pkg, ctx, oracle_mod, first):
    for seed in range(first, first + 20):
        r = random.Random(seed)
        nd = r.choice([2, 2, 3])
        prob = r.choice([CH2, CH2, BIO] if nd == 2 else [CH3, CH3, GROWTH])
        mn = -r.randint(0, 4 if nd == 2 else 3)
        bc = [r.choice([W, PX]) for _ in range(nd)]
        n = []
        for b in bc:
            c = r.randint(2, max(2, r.choice([3, 6, (128 if nd == 2 else 32) >> -mn])))
            n.append((c + (c & 1 if b == PX or mn == 0 else 0)) << -mn)  # a root's and periodic extents are even
        qpo = [0.25, -0.5, 0.75][:prob[2]] if bc[0] == PX and r.random() < 0.5 else None
        g, o = pair(pkg, ctx, oracle_mod, prob, n, mn, bc, qpo, seed)
        g.set_tail_cells(r.choice([2048, 0]))
        calls = []
        for _ in range(5):
            level, ns = r.randint(mn, 0), r.randint(0, 3)
            low = r.randint(mn, level)
            calls.append(r.choice([("set_ghost", level, 0), ("level_relax", level, ns), ("vcycle", level, low, ns),
                                   ("fill_down", r.choice("qf"), level, low), ("copy_q_to_qold", mn, 0),
                                   ("residual_norm", level), ("relax_level_color", level, 1 + ns % 2),
                                   ("time_step", True, 0, low, max(1, ns), 2, 1e-300),
                                   ("multigrid_iterations", 0, low, max(1, ns), 2, 1e-300)]))
            for h in (g, o):
                getattr(h, calls[-1][0])(*calls[-1][1:])
            assert differences(g, o, mn) == [], (seed, n, mn, bc, qpo, calls)
        g.close()
