"""The DMMA GEMM's 32 x 32 tiles and its split of K over a cluster, at tile edges and odd strides."""
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


# below one 64 x 64 tile per SM: unsplit (short K), split in 2 .. 8 (long K), larger tiles split too
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 33, 17), (32, 32, 16), (33, 31, 64), (65, 1, 129), (64, 96, 127),
                                   (32, 96, 1024), (128, 128, 1000), (129, 127, 515), (512, 512, 512), (1000, 30, 260),
                                   (500, 900, 700), (1024, 96, 32)])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("pad,beta,tri", [(0, 0.0, 0), (1, -0.5, 0), (2, 1.0, 1)])
def test_small_products(h, m, n, k, ta, tb, pad, beta, tri):
    import torch
    if tri:
        n = m
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    a = rng.standard_normal((m, k) if ta == "N" else (k, m))
    b = rng.standard_normal((k, n) if tb == "N" else (n, k))
    c = rng.standard_normal((m, n))

    def dev(x):  # column-major with a leading dimension of rows + pad (odd: 8-byte copies)
        t = torch.zeros((x.shape[1], x.shape[0] + pad), dtype=torch.float64, device="cuda")
        t[:, : x.shape[0]] = torch.from_numpy(x.T.copy()).cuda()
        return t
    da, db, dc = dev(a), dev(b), dev(c)
    assert zb.lib().zolo_dgemm_dev(h.ptr, ta.encode(), tb.encode(), m, n, k, -1.0, da.data_ptr(), da.shape[1],
                                   db.data_ptr(), db.shape[1], beta, dc.data_ptr(), dc.shape[1], tri, 0) == 0
    torch.cuda.synchronize()
    got = dc.cpu().numpy()[:, :m].T
    opa, opb = (a if ta == "N" else a.T), (b if tb == "N" else b.T)
    ref = beta * c - opa @ opb
    if tri:
        keep = np.tril(np.ones((m, n), dtype=bool))
        assert np.array_equal(got[~keep], c[~keep])
        got, ref = np.where(keep, got, 0), np.where(keep, ref, 0)
    # any summation order: |error| <= (k + 2) eps (|A| |B| + |beta C|) elementwise, both sides
    bound = 2 * (k + 2) * EPS * (np.abs(opa) @ np.abs(opb) + abs(beta) * np.abs(c))
    assert np.all(np.abs(got - ref) <= bound)
    assert np.all(dc.cpu().numpy()[:, m:] == 0.0)  # the padding rows stay
