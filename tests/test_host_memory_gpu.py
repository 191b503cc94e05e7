"""Host memory of a hierarchy is given back when it is closed."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def rss_mb():
    ctypes.CDLL(None).malloc_trim(0)  # what was freed goes back to the system
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("VmRSS")) / 1024.0


def test_a_closed_hierarchy_leaves_no_work_arrays_behind(pkg, ctx):
    """256x256x128: 8.6 million ghosted cells, so that one array over them of
    four bytes each is 34 MB (and is returned to the system when freed)"""
    def cycle(n):
        h = pkg.Hierarchy(ctx, 3, 2, "ch", [5e-4, 0.02])
        h.build_uniform(n, -2, [2] * 6, [0, 0, 0], [1, 1, 0.5])
        h.commit()
        h.close()
    cycle([64, 64, 32])
    before = rss_mb()
    cycle([256, 256, 128])
    grown = rss_mb() - before
    print("grown by %.0f MB" % grown)
    assert grown < 32
