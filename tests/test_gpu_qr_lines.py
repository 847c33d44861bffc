"""Both sides of the lines at which forming Q and the batched solver's QR and Cholesky change their route
(linalg.cpp: panelwise, kPairBatch)."""
import math

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


# one matrix forms Q panel by panel up to 5e5 entries: 499849, 501264; 499499, 500500; 498015, 500010
@pytest.mark.parametrize("m,n", [(707, 707), (708, 708), (1001, 499), (1001, 500), (7905, 63), (8065, 62)])
def test_one_matrix(h, m, n):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(m * n)
    a = torch.randn((n, m), dtype=torch.float64, device="cuda", generator=g)
    dw = a.clone()
    tau = torch.zeros(n, dtype=torch.float64, device="cuda")
    t = torch.zeros(((n + 31) // 32) * 1024, dtype=torch.float64, device="cuda")
    dq = torch.zeros_like(a)
    lib = zb.lib()
    assert lib.zolo_dgeqrf_dev(h.ptr, m, n, -1, dw.data_ptr(), m, tau.data_ptr(), t.data_ptr()) == 0
    assert lib.zolo_dorgqr_dev(h.ptr, m, n, -1, dw.data_ptr(), m, t.data_ptr(), dq.data_ptr(), m) == 0
    torch.cuda.synchronize()
    q, r = dq.T, torch.triu(dw.T[:n])
    # columnwise backward stable, orthogonal to working accuracy: constants 10 n eps
    assert bool((torch.linalg.norm(q @ r - a.T, dim=0) <= 10 * n * EPS * torch.linalg.norm(a.T, dim=0)).all())
    assert float(torch.linalg.norm(q.T @ q - torch.eye(n, dtype=torch.float64, device="cuda"))) <= 10 * n * EPS


# equal members in one bucket, odd sizes: Cholesky by pairs of leaves up to 16 members; 161 x 157 has stacks of
# 319 x 157, 29 | 30 of them on the sides of 1.5e6 entries (Q), 89 | 90 of 4.5e6 (the factorization)
@pytest.mark.parametrize("m,n,count", [(131, 129, 16), (131, 129, 17), (193, 65, 16), (193, 65, 17), (161, 157, 29),
                                       (161, 157, 30), (161, 157, 89), (161, 157, 90)])
def test_members(h, m, n, count):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + count)
    s = torch.logspace(0, -10, n, dtype=torch.float64, device="cuda")
    u = torch.linalg.qr(torch.randn((count, m, n), dtype=torch.float64, device="cuda", generator=g))[0]
    v = torch.linalg.qr(torch.randn((count, n, n), dtype=torch.float64, device="cuda", generator=g))[0]
    a = (u * s) @ v.transpose(1, 2)
    da = a.transpose(1, 2).contiguous()
    dq = torch.zeros_like(da)
    dh = torch.zeros((count, n, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    info, _ = zb.qdwh_batch_dev(h, [(m, n, da[b].data_ptr(), m, dq[b].data_ptr(), m, dh[b].data_ptr(), n)
                                    for b in range(count)])
    assert all(x == 0 for x in info)
    q = dq.transpose(1, 2)
    tol = max(10 * n * EPS, 1e-14)
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    orth = torch.linalg.norm(q.transpose(1, 2) @ q - eye, dim=(1, 2)) / math.sqrt(n)
    back = torch.linalg.norm(a - q @ dh, dim=(1, 2)) / torch.linalg.norm(a, dim=(1, 2))
    assert float(orth.max()) <= tol and float(back.max()) <= tol
