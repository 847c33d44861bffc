"""The one-launch block reflector (reflect.cu) inside the QR: ragged sizes, odd leading dimensions, the
structured stack, and both sides of the lines between the panelwise and the blocked factorization."""
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


def _run(h, a, pad, m_top):
    import torch
    m, n = a.shape
    ld = m + pad
    dw = torch.full((n, ld), 7.0, dtype=torch.float64, device="cuda")
    dw[:, :m] = torch.from_numpy(a.T.copy()).cuda()
    tau = torch.zeros(n, dtype=torch.float64, device="cuda")
    t = torch.zeros(((n + 31) // 32) * 1024, dtype=torch.float64, device="cuda")
    dq = torch.full((n, ld), 7.0, dtype=torch.float64, device="cuda")
    lib = zb.lib()
    assert lib.zolo_dgeqrf_dev(h.ptr, m, n, m_top, dw.data_ptr(), ld, tau.data_ptr(), t.data_ptr()) == 0
    assert lib.zolo_dorgqr_dev(h.ptr, m, n, m_top, dw.data_ptr(), ld, t.data_ptr(), dq.data_ptr(), ld) == 0
    torch.cuda.synchronize()
    assert bool((dw[:, m:] == 7.0).all()) and bool((dq[:, m:] == 7.0).all())  # the padding rows stay
    return dq.T[:m], torch.triu(dw.T[:n])


# one CTA, clusters of 2 to 16 with ragged rows, one column past a 16-column tile; (1224, 1224) to (2125, 2120)
# straddle 1.5e6 (forming Q) and 4.5e6 (the factorization)
@pytest.mark.parametrize("m,n", [(33, 33), (64, 48), (65, 49), (129, 97), (300, 65), (515, 130), (1030, 161), (2049, 81),
                                 (8190, 65), (1224, 1224), (1226, 1225), (2121, 2120), (2125, 2120)])
@pytest.mark.parametrize("pad", [0, 1])
def test_qr_q(h, m, n, pad):
    import torch
    rng = np.random.default_rng(m + n)
    a = rng.standard_normal((m, n)) * np.logspace(0, -8, n)[None, :]
    q, r = _run(h, a, pad, -1)
    da = torch.from_numpy(a).cuda()
    col = torch.linalg.norm(da, dim=0)
    # columnwise backward stable, orthogonal to working accuracy: constants 10 n eps
    assert bool((torch.linalg.norm(q @ r - da, dim=0) <= 10 * n * EPS * col).all())
    assert float(torch.linalg.norm(q.T @ q - torch.eye(n, dtype=torch.float64, device="cuda"))) <= 10 * n * EPS


@pytest.mark.parametrize("m,n", [(40, 33), (130, 129), (257, 200), (601, 320)])
@pytest.mark.parametrize("pad", [0, 1])
def test_structured(h, m, n, pad):
    import torch
    rng = np.random.default_rng(m * n)
    a = np.vstack([rng.standard_normal((m, n)), 0.3 * np.eye(n)])
    q, r = _run(h, a, pad, m)
    da = torch.from_numpy(a).cuda()
    assert bool((torch.linalg.norm(q @ r - da, dim=0) <= 10 * n * EPS * torch.linalg.norm(da, dim=0)).all())
    assert float(torch.linalg.norm(q.T @ q - torch.eye(n, dtype=torch.float64, device="cuda"))) <= 10 * n * EPS
    assert bool((torch.tril(q[m:], -1) == 0.0).all())
