"""The one-pass smoothing's ring of slots where a CTA runs on from one y-tile
into the next (box.cu k_bx_smooth, SmoothSplit), emulated on the CPU as
test_one_pass_schedule_cpu.py does for one tile a CTA: the ring, its position
and the passes count on across tiles, and the first two planes of a tile are
copied in behind the last barrier of the tile before, while that one's last
plane is still being written back."""
import numpy as np
import pytest

from tests.test_one_pass_schedule_cpu import CPT, NS, NSL, Smem, four_sweeps, newton


class Ring(Smem):
    """with the slots that threads touched since the last barrier"""

    def __init__(self, slot_len):
        super().__init__(NSL * slot_len)
        self.slot_len = slot_len
        self.touched = set()

    def read(self, loc, th, it, lo, hi):
        self.touched.add(lo // self.slot_len)
        return super().read(loc, th, it, lo, hi)

    def write(self, loc, v, th, it, lo, hi):
        self.touched.add(lo // self.slot_len)
        super().write(loc, v, th, it, lo, hi)

    def barrier(self):
        super().barrier()
        self.touched = set()


def smooth(e_in, g, pb, fresh, TY, start):
    """k_bx_smooth over the split start[0], start[1], .. of the line in which
    plane z of tile t is t n2 + z; a row of cells a thread"""
    _, n2, n1, HH = e_in.shape
    R = TY + 2 * NS
    AR, W = R * HH, HH // CPT
    SL = 4 * AR
    out = np.full(e_in.shape, np.nan)
    written = np.zeros(e_in.shape, dtype=np.int64)
    for cta in range(len(start) - 1):
        sm = Ring(SL)
        si = it = 0  # the planes and passes of all tiles so far
        p = start[cta]
        while p < start[cta + 1]:
            tile = p // n2
            y0, z0 = tile * TY, p % n2
            P = min(n2 - z0, start[cta + 1] - p) + 2 * NS
            pending = {}  # slot -> the pass that waits for its copy
            cz, v = {}, {}

            def issue(j, k):
                if fresh or j >= P:
                    return
                assert k not in sm.touched, "a copy into a slot still in use"
                for a in range(4):
                    for r in range(R):
                        loc = k * SL + a * AR + r * HH + np.arange(HH)
                        sm.val[loc] = e_in[a, (z0 - NS + j) % n2, (y0 - NS + r) % n1, :]
                        sm.w_it[loc], sm.w_th[loc] = it - 1, -1
                pending[k] = it0 + j

            def load(s, j, th):
                r, hs = th // W, CPT * (th % W) + np.arange(CPT)
                if s <= j <= P - 1 - s and s <= r <= R - 1 - s:
                    c, zw, yy = (s - 1) & 1, (z0 - NS + j) % n2, (y0 - NS + r) % n1
                    v[(th, s)] = (pb[c, zw, yy, hs], g[c, zw, yy, hs], g[2 + c, zw, yy, hs])

            it0 = it
            issue(0, si % NSL)
            issue(1, (si + 1) % NSL)
            for i in range(P):
                slot = lambda d: (si - d) % NSL
                fw = {}
                for th in range(W * R):
                    r, hc = th // W, CPT * (th % W)
                    for s in range(1, NS + 1):
                        j = i - s
                        if s <= j <= P - 1 - s and s <= r <= R - 1 - s:
                            c, o = (s - 1) & 1, 1 - ((s - 1) & 1)
                            first = (s if s <= 2 else 0) if fresh else 0
                            bb = (c + y0 - NS + r + z0 - NS + j + 1) & 1
                            for d in (s, s + 1, s - 1):
                                assert pending.get(slot(d), -1) <= it, "a slot read while its copy is in flight"
                            base = {d: slot(d) * SL for d in (s - 1, s, s + 1)}

                            def rd(d, loc):
                                return sm.read(base[d] + loc, th, it, base[d], base[d] + SL)
                            sums, xv = [np.zeros(CPT), np.zeros(CPT)], np.zeros(CPT)
                            if first != 1:
                                for var in range(2):
                                    ao = (2 * var + o) * AR + r * HH
                                    cells = ao + hc + np.arange(CPT)
                                    a = cz[(th, s)][var] if j > s else rd(s, cells)
                                    zp = rd(s - 1, cells) if s == 1 else fw[(th, s - 1)][var]
                                    cz.setdefault((th, s), [None, None])[var] = zp
                                    zm, ym, yp = rd(s + 1, cells), rd(s, cells - HH), rd(s, cells + HH)
                                    edge = rd(s, ao + ((hc + CPT) % HH if bb else (hc - 1) % HH))
                                    lft = a if bb else np.concatenate(([edge], a[:-1]))
                                    rgt = np.concatenate((a[1:], [edge])) if bb else a
                                    sums[var] = (lft + rgt + ym + yp) + (zm + zp)
                                if first == 0:
                                    xv = rd(s, c * AR + r * HH + hc + np.arange(CPT))
                            pbv, g0, g1 = v[(th, s)]
                            fw[(th, s)] = newton(pbv, xv, sums[0], sums[1], g0, g1)
                            for var in range(2):
                                sm.write(base[s] + (2 * var + c) * AR + r * HH + hc + np.arange(CPT),
                                         fw[(th, s)][var], th, it, base[s], base[s] + SL)
                        load(s, i + 1 - s, th)
                sm.barrier()
                j = i - NS
                back = NS <= j <= P - 1 - NS
                if back:
                    sm.touched.add(slot(NS))  # other threads may be writing back already
                issue(i + 2, slot(NSL - 2))
                if back:
                    for a in range(4):
                        for rr in range(TY):
                            out[a, z0 - NS + j, y0 + rr, :] = sm.val[slot(NS) * SL + a * AR + (NS + rr) * HH + np.arange(HH)]
                            written[a, z0 - NS + j, y0 + rr, :] += 1
                si += 1
                it += 1
            p += P - 2 * NS
    assert (written == 1).all(), "every output cell written exactly once"
    return out


@pytest.mark.parametrize("fresh", [False, True])
@pytest.mark.parametrize("shape,start", [((4, 24, 8), [0, 12]), ((8, 16, 8), [0, 5, 16]), ((6, 24, 12), [0, 10, 18])])
def test_a_ring_that_runs_on_into_the_next_tile_equals_four_sweeps(shape, start, fresh):
    n2, n1, hh = shape
    rng = np.random.default_rng(n2 * 100 + n1 + hh)
    e = rng.standard_normal((4, n2, n1, hh)) * 1e-2
    g = rng.standard_normal((4, n2, n1, hh)) * 1e-3
    pb = rng.standard_normal((2, n2, n1, hh)) * 0.5
    assert np.array_equal(four_sweeps(e, g, pb, fresh), smooth(e, g, pb, fresh, 8, start))
