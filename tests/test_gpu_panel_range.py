"""Reflectors at the top of the range (qr.cu): columns of norm up to the square root of the largest number."""
import numpy as np
import pytest
import zolo_svd_b200 as zb

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


# norms of 1e154 and, past 6.7e153, (|alpha| + norm)^2 above the largest number; one CTA and a cluster
@pytest.mark.parametrize("norm", [1.0, 6e153, 7e153, 1e154, 1.3e154])
@pytest.mark.parametrize("m", [100, 600])
def test_large_columns(norm, m):
    import torch
    w = 32
    rng = np.random.default_rng(m)
    a = rng.standard_normal((m, w))
    a[np.arange(w), np.arange(w)] = 0.0
    a *= 0.6 / np.linalg.norm(a, axis=0)
    a[np.arange(w), np.arange(w)] = 0.8
    a *= norm
    h = zb.Handle(0)
    da = zb.colmajor_to_device(a)
    tau = torch.empty(w, dtype=torch.float64, device="cuda")
    t = torch.empty(1024, dtype=torch.float64, device="cuda")
    assert zb.lib().zolo_dgeqrf_dev(h.ptr, m, w, -1, da.data_ptr(), m, tau.data_ptr(), t.data_ptr()) == 0
    torch.cuda.synchronize()
    f = zb.device_to_colmajor(da)
    h.close()
    r = np.triu(f[:w]) / norm
    v = np.tril(f, -1)
    v[np.arange(w), np.arange(w)] = 1.0
    tm = t.cpu().numpy().reshape(32, 32).T
    q = np.eye(m, w) - v @ (tm @ v[:w].T)
    # columnwise backward stable, as for columns of norm one
    assert np.all(np.linalg.norm(q @ r - a / norm, axis=0) <= 10 * 32 * EPS)
    assert np.linalg.norm(q.T @ q - np.eye(w)) <= 10 * 32 * EPS
