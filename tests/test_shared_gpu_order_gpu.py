"""Which launches of a hierarchy are made ahead of the previous kernel's end:
those of one whose solves have the GPU to themselves, however many others
there are; none once a solve of it ran beside another's."""
import threading

import pytest

from test_stream_order_gpu import box, cu, edge_types  # noqa: F401 (cu: a fixture)

pytestmark = pytest.mark.gpu


def step(h, first=False):
    h.time_step(first, 0, -6, tol=1e-30, maxvcycles=20, mode="fp64")


def test_many_hierarchies_stepped_in_turn_launch_early(pkg, ctx, cu):  # noqa: F811
    hs = [box(pkg, ctx, (128, 128), -6) for _ in range(12)]
    for h in hs:
        step(h, True)
    kinds = [set(edge_types(cu, h, lambda h=h: h.vcycle(0, -6, 2))) for h in hs]
    for h in hs:
        h.close()
    assert all(1 in k for k in kinds)


def test_solves_side_by_side_take_the_plain_order(pkg, ctx, cu):  # noqa: F811
    """Two threads step two hierarchies until both have seen the other: each
    has at least 200 steps of some 2 ms beside the other's."""
    hs = [box(pkg, ctx, (128, 128), -6) for _ in range(2)]
    start = threading.Barrier(2)
    errors = []

    def work(h):
        try:
            step(h, True)
            start.wait()
            for _ in range(200):
                step(h)
        except Exception as e:  # reported below
            errors.append(e)
    th = [threading.Thread(target=work, args=(h,)) for h in hs]
    for t in th:
        t.start()
    for t in th:
        t.join()
    kinds = [set(edge_types(cu, h, lambda h=h: h.vcycle(0, -6, 2))) for h in hs]
    for h in hs:
        h.close()
    assert not errors
    assert kinds == [{0}, {0}]
