"""Performance cases: what a user of this framework has it compute.

Each case is one pass through the public entry points of the package: a run
of time steps from a given state (put, set_ghost, copy_q_to_qold, time_step,
get, as bench.py and the tests drive them), the same with the mesh rebuilt
before every step (regrid), or the allocation-free residual norm on
caller-owned device buffers.  Both arithmetic modes appear: "fp64" is the
drop-in path, "mixed" the FP32 smoothing inside an FP64 defect-correction
loop.  Sizes are those of bench.py's workloads, the serving stream
(serve.poisson_stream: roots of 32..256 in 2D, 32 and 64 in 3D) and ragged
ones between them.

Ranges (draw): 2D roots of 16..384 cells per side and 3D roots of 16..256,
multiples of 8 that differ by dimension; 1 to 12 time steps; interface width
0.01..0.03; adaptive 2D runs of a 48..96 root with 1 to 3 refinement levels
and growth runs of a 16..32 root with 1 or 2; norms of 2D and 3D patches of
any extent up to 256^3 cells.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

pkg = load_package()

MAXV = 30
_ctx = None


def _context():
    """One context for all hierarchies of a program."""
    global _ctx
    if _ctx is None:
        _ctx = pkg.Context(0)
    return _ctx


def listed():
    return [
        # a small serving request: the smallest root of the stream, where
        # launches and the coarse levels' serial chain are everything
        dict(name="box2d-32-mixed", kind="box", mode="mixed", n0=32, n1=32, n2=1, steps=8, eps=0.02, dt=1e-3, tol=1e-8),
        # the 2D benchmark configuration, mixed and drop-in
        dict(name="box2d-128-mixed", kind="box", mode="mixed", n0=128, n1=128, n2=1, steps=10, eps=0.01, dt=1e-3,
             tol=1e-9),
        dict(name="box2d-128-fp64", kind="box", mode="fp64", n0=128, n1=128, n2=1, steps=10, eps=0.01, dt=1e-3,
             tol=1e-9),
        # the larger 3D serving request, an ordinary 3D run
        dict(name="box3d-64-mixed", kind="box", mode="mixed", n0=64, n1=64, n2=64, steps=5, eps=0.02, dt=5e-4,
             tol=1e-8),
        # the headline 3D benchmark configuration, mixed and drop-in
        dict(name="box3d-256-mixed", kind="box", mode="mixed", n0=256, n1=256, n2=256, steps=4, eps=0.02, dt=5e-4,
             tol=1e-8),
        dict(name="box3d-256-fp64", kind="box", mode="fp64", n0=256, n1=256, n2=256, steps=1, eps=0.02, dt=5e-4,
             tol=1e-8),
        # a ragged 3D domain with walls (Dirichlet faces), as the 3D CH
        # plugin's own boundary conditions are
        dict(name="wall3d-96x64x48-mixed", kind="wall", mode="mixed", n0=96, n1=64, n2=48, steps=3, eps=0.02, dt=5e-4,
             tol=1e-8),
        # the second reference problem on a ragged 2D domain, drop-in only
        dict(name="bio2d-192x128-fp64", kind="bio", mode="fp64", n0=192, n1=128, n2=1, steps=4, eps=0.05, dt=0.1,
             tol=1e-9),
        # the adaptive 2D benchmark configuration: regrid before every step
        dict(name="amr2d-64-mixed", kind="amr", mode="mixed", n0=64, levels=3, steps=8, eps=0.01, dt=1e-3, tol=1e-9),
        dict(name="amr2d-64-fp64", kind="amr", mode="fp64", n0=64, levels=3, steps=4, eps=0.01, dt=1e-3, tol=1e-9),
        # the adaptive 3D growth configuration (three variables)
        dict(name="growth3d-32-mixed", kind="growth", mode="mixed", n0=32, levels=2, steps=3, eps=0.025, dt=0.01,
             tol=1e-8),
        # a host's own convergence test on buffers it keeps
        dict(name="norm3d-160x96x128", kind="norm", mode="fp64", n0=160, n1=96, n2=128, steps=1, eps=0.02, dt=5e-4,
             tol=1.0),
    ]


def draw(rng):
    """One more case of the ranges above."""
    kind = rng.choice(["box", "box", "box", "wall", "bio", "amr", "growth", "norm"])
    logu = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))
    eps = round(rng.uniform(0.01, 0.03), 4)
    if kind == "norm":
        n = [max(3, int(logu(17, 250))) for _ in range(3)]
        if rng.random() < 0.4:
            n = [4 * n[0] + 1, 3 * n[1], 1]
        return dict(kind=kind, mode="fp64", n0=n[0], n1=n[1], n2=n[2], steps=1, eps=eps, dt=5e-4, tol=1.0)
    if kind in ("amr", "growth"):
        if kind == "amr":
            return dict(kind=kind, mode=rng.choice(["mixed", "fp64"]), n0=rng.choice([48, 64, 80, 96]),
                        levels=rng.randint(1, 3), steps=rng.randint(1, 5), eps=round(rng.uniform(0.01, 0.02), 4),
                        dt=1e-3, tol=1e-9)
        return dict(kind=kind, mode=rng.choice(["mixed", "fp64"]), n0=rng.choice([16, 24, 32]),
                    levels=rng.randint(1, 2), steps=rng.randint(1, 3), eps=round(rng.uniform(0.02, 0.03), 4), dt=0.01,
                    tol=1e-8)
    mode = "fp64" if kind == "bio" else rng.choice(["mixed", "mixed", "fp64"])
    if kind == "bio" or rng.random() < 0.5:
        n0 = 8 * round(logu(16, 384) / 8)
        n1 = max(16, 8 * round(n0 * rng.uniform(0.5, 1.0) / 8))
        n = [n0, n1, 1]
        steps = rng.randint(1, 12) if mode == "mixed" else rng.randint(1, 4)
        if kind == "bio":
            return dict(kind=kind, mode=mode, n0=n0, n1=n1, n2=1, steps=steps, eps=0.05, dt=0.1, tol=1e-9)
        return dict(kind=kind, mode=mode, n0=n0, n1=n1, n2=1, steps=steps, eps=eps, dt=1e-3, tol=1e-9)
    top = 256 if kind == "box" else 128
    n0 = 8 * round(logu(16, top) / 8)
    n = [n0] + [max(16, 8 * round(n0 * rng.uniform(0.5, 1.0) / 8)) for _ in range(2)]
    cells = n[0] * n[1] * n[2]
    most = max(1, min(5, (1 << 25) // cells)) if mode == "mixed" else max(1, min(3, (1 << 22) // cells))
    return dict(kind=kind, mode=mode, n0=n[0], n1=n[1], n2=n[2], steps=rng.randint(1, most), eps=eps, dt=5e-4, tol=1e-8)


def _extents(case):
    n = [case["n0"], case["n1"], case["n2"]]
    return [n[0], n[1]] if n[2] == 1 else n


def _minlevel(n, even):
    """Below-root levels while every extent halves: down to even extents of
    at least 2 cells (a periodic box) or to any extent of at least 2."""
    l, n = 0, list(n)
    while l > -9 and all(v % 2 == 0 and v // 2 >= 2 and not (even and (v // 2) % 2) for v in n):
        n = [v // 2 for v in n]
        l -= 1
    return l


def _lap(a, h):
    """Undivided periodic Laplacian over h^2."""
    s = -2.0 * a.dim() * a
    for d in range(a.dim()):
        s = s + torch.roll(a, 1, d) + torch.roll(a, -1, d)
    return s / (h * h)


def _smooth_field(n, seed, mean, amp):
    """A seeded random field on the GPU (float64): mean + amp * U(-1, 1)."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)
    return mean + amp * (2.0 * torch.rand(tuple(n), generator=g, device="cuda", dtype=torch.float64) - 1.0)


def _ghosted(fields):
    """Fields on the interior -> the ghosted Fortran-ordered array (zero ghosts) as a flat tensor."""
    n = tuple(fields[0].shape)
    q = torch.zeros((len(fields),) + tuple(v + 2 for v in reversed(n)), device="cuda", dtype=torch.float64)
    sl = tuple(slice(1, -1) for _ in n)
    for v, f in enumerate(fields):
        q[v][sl] = f.permute(*range(f.dim() - 1, -1, -1))
    return q.reshape(-1)


def _initial(case, seed):
    """phi and mu (or the nutrient) of a uniform run's start."""
    n = _extents(case)
    h = 1.0 / n[0]
    if case["kind"] == "bio":
        # a seeded colony: phi in a noisy disc, nutrient 1
        ax = [(torch.arange(v, device="cuda", dtype=torch.float64) + 0.5) * h for v in n]
        x, y = torch.meshgrid(*ax, indexing="ij")
        r = torch.sqrt((x - 0.5) ** 2 + (y - 0.5 * n[1] * h) ** 2)
        phi = torch.tanh((0.15 - r) / (math.sqrt(2.0) * case["eps"])) + _smooth_field(n, seed, 0.0, 0.02)
        return phi, torch.ones_like(phi)
    phi = _smooth_field(n, seed, 0.1 if len(n) == 3 else 0.0, 0.05)
    mu = phi * phi * phi - phi - case["eps"] ** 2 * _lap(phi, h)
    return phi, mu


class _Run:
    """A uniform run: hierarchy, its start on the host, a buffer for the result."""


def prepare(case, seed):
    s = _Run()
    s.case, s.kind, s.mode = case, case["kind"], case["mode"]
    if s.kind == "norm":
        n = _extents(case)
        s.n, s.h = n, 1.0 / n[0]
        phi, mu = _initial(case, seed)
        s.q = _ghosted([phi, mu])
        old = phi + 1e-3 * _smooth_field(n, seed + 1, 0.0, 1.0)
        s.f = torch.stack([old, -old]).permute(0, *range(len(n), 0, -1)).contiguous().reshape(-1)
        s.out = torch.zeros(1, device="cuda", dtype=torch.float64)
        return s
    if s.kind in ("amr", "growth"):
        nd = 2 if s.kind == "amr" else 3
        nv = 2 if s.kind == "amr" else 3
        n = case["n0"]
        s.minlevel = _minlevel([n] * nd, False)
        prm = [case["dt"], case["eps"]] + ([1.5, 2.0, 0.5, 1.0] if nd == 3 else [])
        bc = [2, 2, 2, 2, 10, 10] if nd == 2 else [10] * 6
        init = (pkg.initial.ch_circle_patch(case["eps"], seed, radius=0.25, noise=0.01) if nd == 2 else
                pkg.initial.growth_sphere(case["eps"], seed, radius=0.1, noise=0.02))
        root = pkg.Hierarchy(_context(), nd, nv, "ch" if nd == 2 else "growth", prm)
        root.build_uniform([n] * nd + [1] * (3 - nd), s.minlevel, bc, [0, 0, 0], [1, 1, 1])
        root.commit()
        root.put(0, "q", init(0, [n] * nd, [1.0 / n] * nd, [0.0] * nd))
        # the mesh of the initial condition, which the first step regrids
        s.start = root.regrid(_regrid_params(case, 0), init)
        root.close()
        return s
    n = _extents(case)
    nd = len(n)
    mx = n + [1] * (3 - nd)
    s.n, s.h = n, 1.0 / n[0]
    s.minlevel = _minlevel(n, s.kind == "box")
    bc = [2] * (2 * nd) + [10] * (6 - 2 * nd) if s.kind == "box" else [10] * 6
    prm = [case["dt"], case["eps"]] + ([1.5, 2.0, 0.5] if s.kind == "bio" else [])
    s.hier = pkg.Hierarchy(_context(), nd, 2, "biogrowth" if s.kind == "bio" else "ch", prm)
    s.hier.build_uniform(mx, s.minlevel, bc, [0, 0, 0], [v / n[0] for v in n] + [1] * (3 - nd))
    s.hier.commit()
    q = _ghosted(_initial(case, seed))
    s.host = torch.empty(q.numel(), dtype=torch.float64, pin_memory=True)
    s.host.copy_(q)
    s.back = torch.empty(q.numel(), dtype=torch.float64, pin_memory=True)
    s.q0, s.q1 = s.host.numpy(), s.back.numpy()
    return s


def _regrid_params(case, step):
    return pkg.regrid_params(case["levels"], tagging="gradient", initial=step == 0, maxside=64,
                             first_id=100000 * (step + 1), ibuffer=1, minimumgridpoints=4, qtolerance=0.25,
                             desiredfillratio=0.9)


def _levels(h, case, nd, nv):
    """The solution of every level 0..levels on the level's own global frame
    (zero where the level has no patch), as a plotting program collects it."""
    out = [np.zeros([case["n0"] << l] * nd + [nv], order="F") for l in range(case["levels"] + 1)]
    for p in h.patch_table():
        if p["level"] < 0:
            continue
        q = h.get(p["id"], "q").reshape([v + 2 for v in p["mx"][:nd]] + [nv], order="F")
        at = tuple(slice(p["mglobal"][2 * d] - 1, p["mglobal"][2 * d + 1]) for d in range(nd))
        out[p["level"]][at] = q[tuple(slice(1, -1) for _ in range(nd))]
    return out


def run(s):
    case = s.case
    if s.kind == "norm":
        pkg.api.ch_residual_norm_noalloc(s.q.data_ptr(), s.f.data_ptr(), len(s.n), s.n, s.h, case["dt"], case["eps"],
                                         s.out.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        return {"norm": s.out}
    cycles = 0
    if s.kind in ("amr", "growth"):
        h = s.start
        for step in range(case["steps"]):
            new = h.regrid(_regrid_params(case, step + 1))
            if h is not s.start:
                h.close()
            h = new
            k, _ = h.time_step(step == 0, h.level_range()[1], s.minlevel, 2, MAXV, case["tol"], mode=s.mode)
            cycles += k
        levels = _levels(h, case, 2 if s.kind == "amr" else 3, 2 if s.kind == "amr" else 3)
        h.close()
        return {"q": levels, "cycles": cycles}
    h = s.hier
    h.put_flat(0, "q", s.q0)
    h.set_ghost(0, 0)
    h.copy_q_to_qold(s.minlevel, 0)
    for step in range(case["steps"]):
        k, _ = h.time_step(step == 0, 0, s.minlevel, 2, MAXV, case["tol"], mode=s.mode)
        cycles += k
    h.get(0, "q", out=s.q1)
    shape = [v + 2 for v in s.n] + [2]
    q = s.q1.reshape(shape, order="F")[tuple(slice(1, -1) for _ in s.n)]
    return {"q": q, "cycles": cycles}


def work(case):
    """Bytes: every step reads the state once and writes it once (FP64, all
    variables).  Operations: of every V-cycle, the four red-black passes over
    every level, the coarse loading and the residual (about 40 operations a
    cell for each pass over a cell's colour pair, 30 for each operator), with
    the V-cycles a step of this problem takes."""
    if case["kind"] == "norm":
        cells = case["n0"] * case["n1"] * case["n2"]
        return {"bytes": 32.0 * cells, "flops": 30.0 * cells}
    if case["kind"] == "amr":  # the refined band around the interface
        cells, nv, cycles, levels = case["n0"] ** 2 + 3.0 * case["n0"] * 2 ** case["levels"] * 4, 2, 7, 4.0 / 3
    elif case["kind"] == "growth":
        cells, nv, cycles, levels = case["n0"] ** 3 * (1.0 + case["levels"]), 3, 6, 8.0 / 7
    else:
        cells, nv = case["n0"] * case["n1"] * case["n2"], 2
        cycles, levels = (5, 8.0 / 7) if case["n2"] > 1 else (9, 4.0 / 3)
    per_cell = 4 * 40 + 2 * 30
    return {"bytes": 16.0 * nv * cells * case["steps"],
            "flops": per_cell * nv / 2 * cells * levels * cycles * case["steps"]}


def exact(case, seed):
    """The converged solution of the same discrete steps in 64 bits, where it
    has a plain form: the norm's formula, and on periodic boxes the implicit
    step solved by a Fourier fixed point."""
    if case["kind"] == "norm":
        s = prepare(case, seed)
        n = s.n
        nd = len(n)
        q = s.q.reshape((2,) + tuple(v + 2 for v in reversed(n)))
        f = s.f.reshape((2,) + tuple(reversed(n)))
        mid = tuple(slice(1, -1) for _ in n)

        def lap(a):
            t = -2.0 * nd * a[mid]
            for d in range(nd):
                for o in (0, 2):
                    t = t + a[tuple(slice(o, o + a.shape[e] - 2) if e == d else slice(1, -1) for e in range(nd))]
            return t

        c0, c1 = case["dt"] / s.h ** 2, case["eps"] ** 2 / s.h ** 2
        r0 = f[0] - (q[0][mid] - c0 * lap(q[1]))
        r1 = f[1] - (q[1][mid] - q[0][mid] ** 3 + c1 * lap(q[0]))
        return {"norm": torch.sqrt(((r0 * r0).sum() + (r1 * r1).sum()) / (2 * r0.numel())).reshape(1)}
    if case["kind"] != "box":
        return None
    n = _extents(case)
    h = 1.0 / n[0]
    c0, c1 = case["dt"] / h ** 2, case["eps"] ** 2 / h ** 2
    phi, mu = _initial(case, seed)
    lam = torch.zeros((1,) * len(n), device="cuda", dtype=torch.float64)
    for d, v in enumerate(n):
        k = torch.arange(v // 2 + 1 if d == len(n) - 1 else v, device="cuda", dtype=torch.float64)
        shape = [1] * len(n)
        shape[d] = -1
        lam = lam + (2.0 * torch.cos(2.0 * math.pi * k / v) - 2.0).reshape(shape)
    for _ in range(case["steps"]):
        old = phi
        oldh = torch.fft.rfftn(old)
        for it in range(400):
            a = 1.5 * float(phi.abs().max()) ** 2
            rhs = oldh + c0 * lam * torch.fft.rfftn(phi * phi * phi - a * phi - old)
            new = torch.fft.irfftn(rhs / (1.0 + c0 * c1 * lam * lam - c0 * a * lam), s=n)
            change = float((new - phi).abs().max())
            phi = new
            if change < 1e-14:
                break
        lap = torch.fft.irfftn(lam * torch.fft.rfftn(phi), s=n)
        mu = phi * phi * phi - old - c1 * lap
    return {"q": torch.stack([phi, mu], dim=-1), "cycles": None}
