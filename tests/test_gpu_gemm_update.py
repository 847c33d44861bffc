"""The DMMA GEMM's short-K updates (C staged in shared memory) and its general tiles, whole and split over K."""
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


# updates: one to sixteen K tiles, ragged last tiles of 1 row, column and K, odd leading dimensions (8-byte
# copies).  General tiles: M = 128 with a long K (split in 8), a wave and a bit, lower triangles
@pytest.mark.parametrize("m,n,k,ta,tb,tri", [
    (1024, 1024, 33, 0, 0, 0), (1217, 897, 48, 0, 0, 0), (1025, 1089, 64, 0, 1, 0), (1089, 1025, 65, 0, 0, 0),
    (1500, 1301, 128, 0, 0, 0), (1409, 1153, 255, 0, 0, 0), (2049, 961, 256, 0, 0, 0), (9700, 64, 64, 0, 0, 0),
    (128, 2100, 3001, 1, 0, 0), (1601, 1555, 300, 0, 1, 0), (777, 1300, 1025, 1, 1, 0), (1281, 1281, 700, 1, 0, 1),
    (2500, 2500, 130, 0, 1, 1)])
@pytest.mark.parametrize("pad,alpha,beta", [(0, -1.0, 1.0), (1, 1.0, -0.5), (0, 0.75, 0.0), (2, -1.0, 2.0)])
def test_products(h, m, n, k, ta, tb, tri, pad, alpha, beta):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k)

    def dev(rows, cols):  # column-major; pad 1: an odd leading dimension, else an even one
        ld = rows + pad
        ld += (ld ^ pad) & 1
        return torch.randn((cols, ld), dtype=torch.float64, device="cuda", generator=g)
    da, db, dc = dev(k if ta else m, m if ta else k), dev(n if tb else k, k if tb else n), dev(m, n)
    a = da[:, : (k if ta else m)].T
    b = db[:, : (n if tb else k)].T
    a, b = (a.T if ta else a), (b.T if tb else b)
    c0 = dc.clone()
    want = alpha * (a @ b) + beta * c0[:, :m].T
    bound = (k + 4) * EPS * (abs(alpha) * (a.abs() @ b.abs()) + abs(beta) * c0[:, :m].T.abs())
    assert zb.lib().zolo_dgemm_dev(h.ptr, b"T" if ta else b"N", b"T" if tb else b"N", m, n, k, alpha, da.data_ptr(),
                                   da.shape[1], db.data_ptr(), db.shape[1], beta, dc.data_ptr(), dc.shape[1], tri,
                                   0) == 0
    torch.cuda.synchronize()
    got = dc[:, :m].T
    mask = torch.ones((m, n), dtype=torch.bool, device="cuda")
    if tri:
        mask = torch.tril(mask)
        assert torch.equal(got[~mask], c0[:, :m].T[~mask])  # the upper triangle is not written
    assert bool((((got - want).abs() <= 2 * bound) | ~mask).all())
    assert torch.equal(dc[:, m:], c0[:, m:])  # nor the rows past m
