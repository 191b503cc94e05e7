"""Which launches of an FP64 V-cycle are made ahead of the previous kernel's
end: none in 3D, those of up to a CTA an SM in 2D."""
import pytest

from test_stream_order_gpu import box, cu, edge_types  # noqa: F401 (cu: a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,mn,expected", [((64, 64, 64), -5, {0}), ((128, 128), -6, {1}), ((512, 512), -8, {0, 1})])
def test_early_launches_of_an_fp64_vcycle(pkg, ctx, cu, n, mn, expected):  # noqa: F811
    h = box(pkg, ctx, n, mn)
    kinds = set(edge_types(cu, h, lambda: h.vcycle(0, mn, 2)))
    h.close()
    assert kinds == expected
