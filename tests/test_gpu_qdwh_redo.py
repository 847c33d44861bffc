"""QDWH when the factorization of a Cholesky-form step fails (ZOLO_OPT_INJECT_CHOL_FAIL): that step alone is done
again, with the QR form; the steps before it stand."""
import math

import numpy as np
import pytest
import zolo_svd_b200 as zb

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


def _qdwh(h, a, m, n, inject):
    import torch
    da = zb.colmajor_to_device(a)
    dq, dh = torch.zeros_like(da), torch.zeros((n, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    h.set_option(zb.OPT_INJECT_CHOL_FAIL, inject)
    h.profile(True)
    h.profile_read(reset=True)
    info = zb.qdwh_dev(h, "N", m, n, 0.0, da.data_ptr(), m, dq.data_ptr(), m, dh.data_ptr(), n, 0, 12, 0)
    panels = h.profile_read(reset=True)["qr_panel"]["launches"]
    h.profile(False)
    h.set_option(zb.OPT_INJECT_CHOL_FAIL, 0)
    assert info == 0
    return zb.device_to_colmajor(dq), zb.device_to_colmajor(dh), h.stats(), panels


# each Cholesky-form step of the solve in turn, the last included; QR panel by panel and (2049 x 1100) in blocks
@pytest.mark.parametrize("m,n,kappa", [(33, 33, 1e3), (300, 260, 1e8), (2049, 1100, 1e10)])
def test_one_step_again(m, n, kappa):
    rng = np.random.default_rng(m + n)
    u, v = (np.linalg.qr(rng.standard_normal(sh))[0] for sh in ((m, n), (n, n)))
    a = (u * np.geomspace(1.0, 1.0 / kappa, n)) @ v.T
    h = zb.Handle(0)
    q0, h0, st0, panels0 = _qdwh(h, a, m, n, 0)
    steps = [k for k, b in enumerate(st0["branches"]) if b == "CH"]
    assert st0["info"] == 0 and len(steps) >= 2
    for k in steps:
        q1, h1, st1, panels1 = _qdwh(h, a, m, n, k + 1)
        assert st1["info"] == 1000000
        assert st1["branches"] == [("QR" if i == k else b) for i, b in enumerate(st0["branches"])]
        assert list(st1["con"]) == list(st0["con"])
        assert list(st1["err"])[:k] == list(st0["err"])[:k]  # the same bits
        assert panels1 - panels0 == (n + 31) // 32
        # backward error and orthogonality of the repository's solves, 10 n eps
        assert np.linalg.norm(a - q1 @ h1) / np.linalg.norm(a) <= 10 * n * EPS
        assert np.linalg.norm(q1.T @ q1 - np.eye(n)) / math.sqrt(n) <= 10 * n * EPS
    again = _qdwh(h, a, m, n, 0)
    h.close()
    assert np.array_equal(again[0], q0) and np.array_equal(again[1], h0)


def test_bound_past_one():
    """The lower bound of a single column is 1 up to rounding; past 1 it has no weights (not a number), and the
    iteration ends after its first step as at any other converged L."""
    import torch
    hd = zb.Handle(0)
    rng = np.random.default_rng(5)
    past = 0
    for _ in range(24):
        a = rng.standard_normal((2, 1))
        da = zb.colmajor_to_device(a)
        dq, dh = torch.zeros_like(da), torch.zeros((1, 1), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert zb.qdwh_dev(hd, "N", 2, 1, 0.0, da.data_ptr(), 2, dq.data_ptr(), 2, dh.data_ptr(), 1, 0, 12, 0) == 0
        st = hd.stats()
        past += st["beta"] > 1.0
        assert st["iterations"] == 1
    hd.close()
    assert past > 0
