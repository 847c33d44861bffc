"""Products of a long K over few tiles of C (gemm.cu, plan_gemm): K is split over several clusters a tile, whose
sums go through scratch."""
import pytest
import zolo_svd_b200 as zb

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


@pytest.fixture(scope="module")
def h():
    hd = zb.Handle(0)
    yield hd
    hd.close()


def _check(h, ta, tb, m, n, k, alpha, beta, tri, pad=0):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(m * 7 + n * 3 + k)

    def mat(r, c):  # column-major r x c with leading dimension r + pad
        return torch.randn((c, r + pad), dtype=torch.float64, device="cuda", generator=g)

    a, b, c = mat(*((k, m) if ta == b"T" else (m, k))), mat(*((n, k) if tb == b"T" else (k, n))), mat(m, n)
    av, bv = (x[:, :x.shape[1] - pad].T for x in (a, b))
    av, bv = av.T if ta == b"T" else av, bv.T if tb == b"T" else bv
    c0 = c.clone()
    rc = zb.lib().zolo_dgemm_dev(h.ptr, ta, tb, m, n, k, alpha, a.data_ptr(), a.shape[1], b.data_ptr(), b.shape[1],
                                 beta, c.data_ptr(), c.shape[1], tri, 0)
    assert rc == 0
    got, old = c[:, :m].T, c0[:, :m].T
    want = alpha * (av @ bv) + beta * old
    # |error| <= (K + 2) eps |alpha| |op(A)| |op(B)| + 2 eps |beta C|, twice for the reference's own
    bound = 2 * EPS * ((k + 2) * abs(alpha) * (av.abs() @ bv.abs()) + 2 * abs(beta) * old.abs())
    if tri:
        low = torch.tril(torch.ones_like(want, dtype=torch.bool))
        assert bool(((got - want).abs() <= bound)[low].all())
        assert torch.equal(got[~low], old[~low])
    else:
        assert bool(((got - want).abs() <= bound).all())
    if pad:
        assert torch.equal(c[:, m:], c0[:, m:])


# K on both sides of 2048, 4096 and 16384 (kt = 128, 256, 1024) and ragged, with outputs of one tile and up to one
# tile an SM: every tile shape and number of groups; the last slices of a ragged K are short or empty
@pytest.mark.parametrize("k", [2032, 2033, 2049, 4097, 8191, 16385])
@pytest.mark.parametrize("m,n", [(1, 1), (32, 32), (33, 31), (32, 2049), (17, 4100), (65, 63), (130, 700), (513, 64),
                                 (1025, 129), (6145, 64)])
def test_shapes(h, m, n, k):
    _check(h, b"T", b"N", m, n, k, 1.0, 0.0, 0)


@pytest.mark.parametrize("ta", [b"N", b"T"])
@pytest.mark.parametrize("tb", [b"N", b"T"])
@pytest.mark.parametrize("pad", [0, 1, 2])
def test_forms(h, ta, tb, pad):
    _check(h, ta, tb, 96, 160, 5000, -0.75, 1.5, 0, pad)


@pytest.mark.parametrize("n", [1, 31, 64, 130, 257, 384, 513, 769])
@pytest.mark.parametrize("k", [2047, 4100, 20001])
def test_lower_triangle(h, n, k):
    _check(h, b"T", b"N", n, n, k, 2.0, -1.0, 1)


def test_tall_solve(h):
    """Every product of a tall solve has a long K."""
    import torch
    m, n = 60001, 48
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    u = torch.linalg.qr(torch.randn((m, n), dtype=torch.float64, device="cuda", generator=g))[0]
    v = torch.linalg.qr(torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g))[0]
    a = (u * torch.logspace(0, -8, n, dtype=torch.float64, device="cuda")) @ v.T
    da = a.T.contiguous()
    dq, dh = torch.zeros_like(da), torch.zeros((n, n), dtype=torch.float64, device="cuda")
    res = []
    for _ in range(2):
        assert zb.qdwh_dev(h, "N", m, n, 0.0, da.data_ptr(), m, dq.data_ptr(), m, dh.data_ptr(), n, 0, 12, 0) == 0
        res.append((dq.clone(), dh.clone()))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    q, hh = dq.T, dh.T
    assert float(torch.linalg.norm(a - q @ hh) / torch.linalg.norm(a)) <= 10 * n * EPS
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    assert float(torch.linalg.norm(q.T @ q - eye)) <= 10 * n * EPS


def test_uses_the_gpu(h):
    """32 x 32 x 200000 reads 102 MB: about 60 us; in one cluster of 8 CTAs it took 700.  Against twelve copies of the
    bytes it reads (about 35 us each way)."""
    import torch
    k, n = 200000, 32
    a = torch.randn((2 * n, k), dtype=torch.float64, device="cuda")
    b, c = torch.empty_like(a), torch.zeros((n, n), dtype=torch.float64, device="cuda")

    def best(f):
        t = []
        for _ in range(20):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            f()
            e1.record()
            torch.cuda.synchronize()
            t.append(e0.elapsed_time(e1))
        return min(t)

    def product():
        assert zb.lib().zolo_dgemm_dev(h.ptr, b"T", b"N", n, n, k, 1.0, a[:n].data_ptr(), k, a[n:].data_ptr(), k, 0.0,
                                       c.data_ptr(), n, 0, 0) == 0

    h.set_stream(torch.cuda.current_stream().cuda_stream)
    copies = best(lambda: [b.copy_(a) for _ in range(12)])
    assert best(product) <= copies
