"""Triangular inverse by levels of block pairs, and the Cholesky-form step that applies it."""
import numpy as np
import pytest
import zolo_svd_b200 as zb
from oracle import zolo_oracle as zo

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


@pytest.fixture(scope="module")
def h():
    hd = zb.Handle(0)
    yield hd
    hd.close()


# one leaf, full pairs at every level, a ragged last pair of 1 row, one shorter than its level, odd leading dimensions
@pytest.mark.parametrize("n,pad", [(64, 0), (65, 0), (128, 1), (129, 0), (192, 0), (193, 2), (256, 0), (320, 1),
                                   (520, 0), (576, 0), (701, 0), (1024, 0)])
def test_inverse_of_factor(h, n, pad):
    import torch
    rng = np.random.default_rng(n)
    l = np.tril(rng.standard_normal((n, n))) / np.sqrt(n) + 4.0 * np.eye(n)
    ld = n + pad
    big = np.full((ld, n), np.nan)  # the padding rows and L's upper triangle are not read as L
    big[:n] = l + np.triu(rng.standard_normal((n, n)), 1)
    dl = zb.colmajor_to_device(big)
    dy = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
    assert zb.lib().zolo_dtrtri_dev(h.ptr, n, dl.data_ptr(), ld, dy.data_ptr(), ld) == 0
    y = dy.cpu().numpy().T[:n]
    assert np.all(np.triu(y, 1) == 0.0)
    # residuals of an inverse built from products: n eps ||L|| ||L^{-1}||
    bound = n * EPS * np.linalg.norm(l, 2) * np.linalg.norm(np.linalg.inv(l), 2)
    assert np.linalg.norm(y @ l - np.eye(n), 2) <= bound
    assert np.linalg.norm(l @ y - np.eye(n), 2) <= bound


# all steps in Cholesky form (kappa small), solved from the right and (SYM = 'S') from the left
@pytest.mark.parametrize("sym", ["N", "S"])
@pytest.mark.parametrize("n", [1, 33, 64, 65, 130, 257])
def test_qdwh_cholesky_steps(h, n, sym):
    import torch
    s = np.linspace(1.0, 2.0, n)
    rng = np.random.default_rng(n)
    u, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (u * (s * np.where(np.arange(n) % 2, -1.0, 1.0))[None, :]) @ u.T
    a = 0.5 * (a + a.T)
    da = zb.colmajor_to_device(a)
    dq, dh = torch.zeros_like(da), torch.zeros_like(da)
    zb.qdwh_dev(h, sym, n, n, 0.0, da.data_ptr(), n, dq.data_ptr(), n, dh.data_ptr(), n, 0, 12, 0)
    q, hh = zb.device_to_colmajor(dq), zb.device_to_colmajor(dh)
    assert zo.orthogonality(q) <= 10 * n * EPS + 4 * EPS
    assert zo.backward_error(a, q, hh) <= 10 * n * EPS + 4 * EPS


# two leaves in one launch: one row to a full second leaf, and the levels above it; m > n, so no left solve
@pytest.mark.parametrize("n", [66, 79, 80, 81, 96, 113, 127, 128, 129, 191, 193, 256, 385])
def test_qdwh_paired_leaves(h, n):
    import torch
    m = n + 13
    rng = np.random.default_rng(n)
    u, _ = np.linalg.qr(rng.standard_normal((m, n)))
    v, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (u * np.geomspace(1.0, 0.02, n)[None, :]) @ v.T
    da = zb.colmajor_to_device(a)
    dq, dh = torch.zeros_like(da), torch.zeros((n, n), dtype=torch.float64, device="cuda")
    zb.qdwh_dev(h, "N", m, n, 0.0, da.data_ptr(), m, dq.data_ptr(), m, dh.data_ptr(), n, 0, 12, 0)
    assert h.stats()["chol_iterations"] >= 2
    q, hh = zb.device_to_colmajor(dq), zb.device_to_colmajor(dh)
    assert zo.orthogonality(q) <= 10 * n * EPS
    assert zo.backward_error(a, q, hh) <= 10 * n * EPS
    # the polar factor is determined to kappa eps
    assert np.linalg.norm(q - u @ v.T) <= 10 * n * EPS * 50
