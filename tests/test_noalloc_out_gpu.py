"""Where bsamg_ch_residual_norm_noalloc may write its result: any address of
device memory, as a copy reaches it, whether or not a kernel can store a
double there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 4, 8, 1, 13])
def test_norm_at_any_address(pkg, ctx, offset):
    torch = pytest.importorskip("torch")
    n = [32, 10, 6]
    h = pkg.Hierarchy(ctx, 3, 2, "ch", [1e-3, 0.01])
    h.build_uniform(n, 0, [2, 2, 2, 2, 10, 10], [0, 0, 0], [1, 10 / 32, 6 / 32])
    h.commit()
    rng = np.random.default_rng(4)
    for f in ("q", "f"):
        h.put(0, f, rng.uniform(-1, 1, size=h.field_size(0, f)))
    q, f = (torch.from_numpy(h.get(0, x)).cuda() for x in ("q", "f"))
    out = torch.full((32,), 255, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    pkg.api.ch_residual_norm_noalloc(q.data_ptr(), f.data_ptr(), 3, n, 1.0 / 32, 1e-3, 0.01, out.data_ptr() + offset)
    torch.cuda.synchronize()
    b = out.cpu().numpy().tobytes()
    assert np.frombuffer(b[offset:offset + 8])[0] == h.residual_norm(0)
    assert set(b[:offset] + b[offset + 8:]) == {255}
    h.close()
