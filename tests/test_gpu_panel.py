"""The register-resident Householder panel (qr.cu) at the edges of its row chunks and cluster sizes."""
import numpy as np
import pytest
import zolo_svd_b200 as zb

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


@pytest.fixture(scope="module")
def h():
    hd = zb.Handle(0)
    yield hd
    hd.close()


# one CTA (up to 256 rows), 4, 8 and 16 CTAs, one row either side of every capacity, the largest
# register panel (8192 rows) and the first one past it; narrow panels and a zero column
@pytest.mark.parametrize("m", [1, 2, 31, 33, 127, 128, 129, 255, 257, 512, 513, 1023, 1025, 2049, 4097, 8191, 8192, 8193])
@pytest.mark.parametrize("w", [1, 7, 32])
@pytest.mark.parametrize("zero", [False, True])
def test_panel(h, m, w, zero):
    import torch
    if w > m:
        pytest.skip("panel wider than its rows")
    rng = np.random.default_rng(m * 100 + w)
    a = rng.standard_normal((m, w)) * np.logspace(0, -6, w)[None, :]
    if zero:
        a[:, w // 2] = 0.0
    da = zb.colmajor_to_device(a)
    tau = torch.empty(w, dtype=torch.float64, device="cuda")
    t = torch.empty(1024, dtype=torch.float64, device="cuda")
    assert zb.lib().zolo_dgeqrf_dev(h.ptr, m, w, -1, da.data_ptr(), m, tau.data_ptr(), t.data_ptr()) == 0
    torch.cuda.synchronize()
    f = zb.device_to_colmajor(da)
    r = np.triu(f[:w])
    v = np.tril(f, -1)
    v[np.arange(w), np.arange(w)] = 1.0
    tm = t.cpu().numpy().reshape(32, 32).T
    assert np.all(tm[np.tril_indices(32, -1)] == 0.0) and np.all(tm[:, w:] == 0.0)
    assert np.array_equal(np.diag(tm)[:w], tau.cpu().numpy())
    q = np.eye(m, w) - v @ (tm[:w, :w] @ v[:w].T)
    # Householder QR is columnwise backward stable: ||(QR - A)_j|| <= c w eps ||a_j||; c = 10
    col = np.linalg.norm(a, axis=0)
    assert np.all(np.linalg.norm(q @ r - a, axis=0) <= 10 * 32 * EPS * col)
    assert np.linalg.norm(q.T @ q - np.eye(w)) <= 10 * 32 * EPS
