"""A zero or non-finite matrix is refused before the QR of its bounds, which would be for nothing."""
import numpy as np
import pytest
import zolo_svd_b200 as zb

pytestmark = pytest.mark.gpu


# panel by panel, in blocks, and past the register panels; the launches of one panel against those of the whole QR
@pytest.mark.parametrize("m,n", [(200, 33), (1024, 1024), (4200, 1500), (8300, 300), (8300, 96)])
@pytest.mark.parametrize("bad", [0.0, np.nan, np.inf])
def test_unusable_matrix(m, n, bad):
    import torch
    h = zb.Handle(0)
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n)
    good = torch.randn((n, m), dtype=torch.float64, device="cuda", generator=g)
    a = torch.zeros_like(good)
    if bad != 0.0:
        a.copy_(good)
        a[n // 2, m - 1] = bad
    q, hh = torch.zeros_like(good), torch.zeros((n, n), dtype=torch.float64, device="cuda")

    def qdwh(x):
        return zb.lib().zolo_qdwh_dev(h.ptr, b"N", m, n, 0.0, x.data_ptr(), m, q.data_ptr(), m, hh.data_ptr(), n, 0,
                                      12, 0)

    assert qdwh(good) == 0
    q0 = q.clone()
    assert qdwh(a) == 1
    st = h.stats()
    assert st["info"] == 1 and st["launches"] <= 12
    assert st["alpha"] == 0.0 if bad == 0.0 else not np.isfinite(st["alpha"])
    assert qdwh(good) == 0 and torch.equal(q, q0)
    h.close()
