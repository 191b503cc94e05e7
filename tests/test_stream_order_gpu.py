"""What a call leaves on its hierarchy's stream."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cu():
    L = ctypes.CDLL("libcuda.so.1")
    P, Z = ctypes.c_void_p, ctypes.POINTER(ctypes.c_size_t)
    L.cuStreamQuery.argtypes = [P]
    L.cuStreamBeginCapture_v2.argtypes = [P, ctypes.c_int]
    L.cuStreamEndCapture.argtypes = [P, ctypes.POINTER(P)]
    L.cuGraphGetEdges_v2.argtypes = [P, P, P, P, Z]
    L.cuGraphDestroy.argtypes = [P]
    return L


def edge_types(cu, h, call):
    """the kinds of the dependencies (0 full, 1 programmatic) among the
    launches `call` makes, captured instead of run"""
    call()  # plans are made by the first call
    h.sync()
    g, n = ctypes.c_void_p(), ctypes.c_size_t()
    assert cu.cuStreamBeginCapture_v2(h.stream(), 2) == 0
    try:
        call()
    finally:
        rc = cu.cuStreamEndCapture(h.stream(), ctypes.byref(g))
    assert rc == 0
    assert cu.cuGraphGetEdges_v2(g, None, None, None, ctypes.byref(n)) == 0
    a, b = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)()
    data = (ctypes.c_ubyte * (8 * n.value))()  # from_port, to_port, type, 5 reserved
    assert cu.cuGraphGetEdges_v2(g, a, b, data, ctypes.byref(n)) == 0
    assert cu.cuGraphDestroy(g) == 0
    return [data[8 * x + 2] for x in range(n.value)]


def box(pkg, ctx, n, minlevel):
    nd = len(n)
    h = pkg.Hierarchy(ctx, nd, 2, "ch", [5e-4, 0.02])
    h.build_uniform(list(n) + [1] * (3 - nd), minlevel, [2] * (2 * nd) + [10] * (6 - 2 * nd), [0, 0, 0], [1, 1, 1])
    h.commit()
    h.seed_spinodal(0, 3)
    return h


def test_raised_tail_cells_keep_the_plain_launch_order(pkg, ctx, cu):
    """128^2: two levels of launches above the cluster's V-cycle"""
    h = box(pkg, ctx, (128, 128), -6)
    early = edge_types(cu, h, lambda: h.vcycle(0, -6, 2))
    h.set_tail_cells(16384)
    plain = edge_types(cu, h, lambda: h.vcycle(0, -6, 2))
    h.close()
    assert len(plain) == len(early) > 8
    assert 1 in early and set(plain) == {0}


def test_a_step_is_finished_when_the_call_returns(pkg, ctx, cu):
    """FillDown of q and f below level 0 included (some 100 us of kernels at 160^3)"""
    h = box(pkg, ctx, (160, 160, 160), -4)
    for s in range(3):
        h.time_step(s == 0, 0, -4, tol=1e-30, maxvcycles=1, mode="fp64")
        assert cu.cuStreamQuery(h.stream()) == 0
    h.close()
