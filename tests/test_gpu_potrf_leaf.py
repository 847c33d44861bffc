"""The 64 x 64 Cholesky leaf and its inverse (potrf.cu) at the edges of its 16 x 16 blocks."""
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


def _spd(n, kappa, seed):
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    return (q * np.geomspace(1.0, 1.0 / kappa, n)[None, :]) @ q.T


# one leaf from 1 to 64 rows around every multiple of 16, and two leaves with a ragged second one
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 47, 49, 63, 64, 65, 79, 81, 127])
@pytest.mark.parametrize("kappa", [1e2, 1e6])
def test_leaf_factor_and_inverse(h, n, kappa):
    import torch
    a = _spd(n, kappa, n)
    a = 0.5 * (a + a.T)
    da = zb.colmajor_to_device(a)
    assert zb.lib().zolo_dpotrf_dev(h.ptr, n, da.data_ptr(), n) == 0
    torch.cuda.synchronize()
    l = np.tril(zb.device_to_colmajor(da))
    # backward error of Cholesky n eps; the products with 16 x 16 inverses add their condition, sqrt(kappa) at most
    assert np.linalg.norm(l @ l.T - a) <= 10 * n * EPS * np.linalg.norm(a) * max(1.0, kappa ** 0.25)
    dl, dy = zb.colmajor_to_device(l), torch.zeros((n, n), dtype=torch.float64, device="cuda")
    assert zb.lib().zolo_dtrtri_dev(h.ptr, n, dl.data_ptr(), n, dy.data_ptr(), n) == 0
    torch.cuda.synchronize()
    y = zb.device_to_colmajor(dy)
    assert np.all(np.triu(y, 1) == 0.0)
    # left and right residuals of an inverse formed from block products: n eps ||L|| ||L^-1|| (sqrt(kappa))
    assert np.linalg.norm(y @ l - np.eye(n)) <= 10 * n * EPS * np.sqrt(kappa) * np.sqrt(n)


@pytest.mark.parametrize("n,bad", [(1, 0), (16, 15), (17, 16), (40, 0), (64, 33), (64, 63), (100, 70)])
def test_leaf_info(h, n, bad):
    a = np.eye(n)
    a[bad, bad] = -1.0
    da = zb.colmajor_to_device(a)
    assert zb.lib().zolo_dpotrf_dev(h.ptr, n, da.data_ptr(), n) == bad + 1
