"""Zolo-PD's default form where its Cholesky-form iterations start at a large CON: the factors of the shifted Gram
matrices are then too ill-conditioned for products with their inverses."""
import math

import pytest
import zolo_svd_b200 as zb

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


# CON of the first Cholesky-form iteration: 236, 777, 343, 93, 75 (polar.cpp takes products up to 12).  With
# substitution the backward error is 13 to 16 eps for each of them; three times that is allowed
@pytest.mark.parametrize("m,n,kappa,rk,mixed", [(2400, 2304, 1e15, 8, 1), (2400, 2304, 1e14, 3, 1),
                                                (700, 600, 10 ** 14.5, 3, 0), (2400, 2304, 10 ** 14.5, 6, 1),
                                                (2400, 2304, 10 ** 14.5, 8, 1)])
def test_backward_error(m, n, kappa, rk, mixed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(int(kappa) % 1000 + n)

    def haar(a, b):
        q, r = torch.linalg.qr(torch.randn(a, b, dtype=torch.float64, device="cuda", generator=g))
        return q * torch.sign(torch.diagonal(r))[None, :]

    s = torch.logspace(0, -math.log10(kappa), n, dtype=torch.float64, device="cuda")
    a = (haar(m, n) * s) @ haar(n, n).T
    da = a.T.contiguous()
    dq = torch.empty_like(da)
    dh = torch.empty((n, n), dtype=torch.float64, device="cuda")
    h = zb.Handle(0)
    h.set_option(zb.OPT_MIXED, mixed)
    al, be, _ = zb.bounds_dev(h, m, n, da.data_ptr(), m, mode=1)
    assert zb.pzolopd1_dev(h, "N", rk, m, n, al, be, da.data_ptr(), m, dq.data_ptr(), m, dh.data_ptr(), n) == 0
    st = h.stats()
    h.close()
    assert st["branches"][:2] == ["QR", "CH"] and list(st["con"])[1] > 12.0
    assert float(torch.linalg.norm(a - dq.T @ dh) / torch.linalg.norm(a)) <= 48 * EPS


# two terms: the Cholesky-form iterations start at a CON of about 5 and 31, one on each side of 12
@pytest.mark.parametrize("kappa,products", [(1e3, True), (1e7, False)])
def test_left_form(kappa, products):
    """SYM = 'S' solves from the left, in both routes of the Cholesky-form iteration."""
    import torch
    n = 333
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    v = torch.linalg.qr(torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g))[0]
    s = torch.logspace(0, -math.log10(kappa), n, dtype=torch.float64, device="cuda")
    s[::2] *= -1.0
    a = (v * s) @ v.T
    a = 0.5 * (a + a.T)
    da = a.contiguous()
    dq, dh = torch.empty_like(da), torch.empty_like(da)
    h = zb.Handle(0)
    al, be, _ = zb.bounds_dev(h, n, n, da.data_ptr(), n, mode=1)
    assert zb.pzolopd1_dev(h, "S", 2, n, n, al, be, da.data_ptr(), n, dq.data_ptr(), n, dh.data_ptr(), n) == 0
    st = h.stats()
    h.close()
    first = [c for c, b in zip(st["con"], st["branches"]) if b == "CH"][0]
    assert (first <= 12.0) == products
    q, hh = dq.T, dh.T
    # the polar factor is determined to eps kappa; A - Q H to eps whatever kappa is
    exact = (v * torch.sign(s)) @ v.T
    assert float(torch.linalg.norm(q - exact) / math.sqrt(n)) <= 100 * n * EPS * kappa
    assert float(torch.linalg.norm(a - q @ hh) / torch.linalg.norm(a)) <= 10 * n * EPS
