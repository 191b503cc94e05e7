"""A plugin whose operator reads diagonal neighbours (tests/plugins/corners.cu,
linked into a build of its own): the coarse V-cycle gives the same bits
whether its operations are launches or not, and the residuals it stores are
those of the plugin's operator on the ghosts of SetGhost."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import numpy as np
import __graft_entry__ as ge
pkg = ge.load_package()
ctx = pkg.Context(0)
for n, mn, bc in (((48, 32), -2, (2, 10)), ((96, 96), -3, (10, 10)), ((16, 12, 8), -1, (10, 2, 10))):
    nd = len(n)
    got = []
    for tail in (2048, 0):
        h = pkg.Hierarchy(ctx, nd, 2, "corners", [2e-4, 0.5])
        h.build_uniform(list(n) + [1] * (3 - nd), mn, [b for b in bc for _ in range(2)] + [10] * (6 - 2 * nd),
                        [0, 0, 0], [v / n[0] for v in n] + [1] * (3 - nd))
        h.commit()
        h.set_tail_cells(tail)
        rng = np.random.default_rng(nd)
        for f in ("q", "f"):
            h.put(0, f, rng.uniform(-1, 1, size=h.field_size(0, f)))
        h.set_ghost(0, 0)
        for _ in range(2):
            h.vcycle(0, mn, 2)
        got.append([h.get(p, f) for p in range(1 - mn) for f in ("q", "qc", "f", "rf")])
        h.close()
    print(n, sum(int(np.sum(a != b)) for a, b in zip(*got)))
ctx.close()
"""


def test_operator_with_diagonal_neighbours():
    import __graft_entry__ as ge
    lib = os.path.join(ROOT, "bsam1.2_gb300", "_build", "libbsamg_corners.so")
    env = dict(os.environ, BSAMG_LIBRARY=ge._load_build_module().build(
        extra_plugins=[os.path.join(ROOT, "tests", "plugins", "corners.cu")], lib=lib))
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = r.stdout.strip().splitlines()
    assert len(rows) == 3 and all(row.endswith(") 0") for row in rows), rows
