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


# blocks of 128 columns, the last one with one to four panels and a ragged last panel (its T by pairs of panels)
@pytest.mark.parametrize("w", [1, 31, 32, 33, 64, 65, 96, 97, 127, 128])
def test_block_t(h, w):
    import torch
    m, n = 8192, 640 + w
    g = torch.Generator(device="cuda")
    g.manual_seed(w)
    da = torch.randn((m, n), dtype=torch.float64, device="cuda", generator=g)
    q, r = _run(h, da.cpu().numpy(), 0, -1)
    assert bool((torch.linalg.norm(q @ r - da, dim=0) <= 10 * n * EPS * torch.linalg.norm(da, dim=0)).all())
    assert float(torch.linalg.norm(q.T @ q - torch.eye(n, dtype=torch.float64, device="cuda"))) <= 10 * n * EPS


# the mixed form applies Q in blocks of 512 columns: one block, one and a ragged rest, two
@pytest.mark.parametrize("n", [300, 511, 513, 640, 700, 1024, 1100])
def test_wide_blocks(n):
    import torch
    m = n + 37
    hd = zb.Handle(0)
    for o in (zb.OPT_NS_FINISH, zb.OPT_CHOL_INVERSE, zb.OPT_BETA_FROB, zb.OPT_TERM_PLAN, zb.OPT_MIXED):
        hd.set_option(o, 1)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    a = torch.randn((m, n), dtype=torch.float64, device="cuda", generator=g)
    da = a.T.contiguous()
    dq, dh = torch.zeros_like(da), torch.zeros((n, n), dtype=torch.float64, device="cuda")
    zb.polar_dev(hd, 8, m, n, da.data_ptr(), m, dq.data_ptr(), m, dh.data_ptr(), n)
    q, hh = dq.T, dh.T
    assert float(torch.linalg.norm(q.T @ q - torch.eye(n, dtype=torch.float64, device="cuda"))) <= 10 * n * EPS
    assert float(torch.linalg.norm(q @ hh - a) / torch.linalg.norm(a)) <= 10 * n * EPS
    hd.close()
