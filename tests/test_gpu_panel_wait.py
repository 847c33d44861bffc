"""A wait between the thread blocks of a Householder panel that runs out (ZOLO_OPT_PANEL_WAIT): the call says so,
the kernel has received everything sent to it before it ends, and the handle goes on working."""
import numpy as np
import pytest
import zolo_svd_b200 as zb

pytestmark = pytest.mark.gpu
WAIT_RAN_OUT = -2911


@pytest.fixture()
def h():
    hd = zb.Handle(0)
    yield hd
    hd.close()


def _geqrf(h, a):
    import torch
    m, n = a.shape
    da = zb.colmajor_to_device(a)
    tau = torch.zeros(n, dtype=torch.float64, device="cuda")
    t = torch.zeros((n + 31) // 32 * 1024, dtype=torch.float64, device="cuda")
    info = zb.lib().zolo_dgeqrf_dev(h.ptr, m, n, -1, da.data_ptr(), m, tau.data_ptr(), t.data_ptr())
    torch.cuda.synchronize()
    return info, zb.device_to_colmajor(da), t.cpu().numpy()


# clusters of 4, 8 and 16 blocks, ragged rows, one column to two panels
@pytest.mark.parametrize("m", [300, 513, 1025, 2049, 4097, 8192])
@pytest.mark.parametrize("w", [1, 2, 3, 31, 32, 64])
def test_no_wait_at_all(h, m, w):
    assert zb.lib().zolo_panel_cluster_size(m, w) > 1
    a = np.random.default_rng(m + w).standard_normal((m, w))
    h.set_option(zb.OPT_PANEL_WAIT, 0)
    good = _geqrf(h, a)
    assert good[0] == 0
    h.set_option(zb.OPT_PANEL_WAIT, -1)
    assert _geqrf(h, a)[0] == WAIT_RAN_OUT
    h.set_option(zb.OPT_PANEL_WAIT, 0)
    again = _geqrf(h, a)
    assert again[0] == 0 and np.array_equal(again[1], good[1]) and np.array_equal(again[2], good[2])


# limits around the time that an exchange takes: blocks give up at the same or at neighbouring columns, or none does
@pytest.mark.parametrize("m", [513, 1025, 8192])
@pytest.mark.parametrize("limit", [0, 1, 100, 200, 400, 600, 800, 1000, 1500, 3000])
def test_short_waits(h, m, limit):
    a = np.random.default_rng(m).standard_normal((m, 32))
    good = _geqrf(h, a)
    assert good[0] == 0
    for _ in range(5):
        h.set_option(zb.OPT_PANEL_WAIT, limit)
        info, f, t = _geqrf(h, a)
        assert info in (0, WAIT_RAN_OUT)
        if info == 0:
            assert np.array_equal(f, good[1]) and np.array_equal(t, good[2])
        else:
            assert limit > 0
        h.set_option(zb.OPT_PANEL_WAIT, 0)
        assert _geqrf(h, a)[0] == 0


def test_whole_solves_report_it(h):
    import torch
    m, n = 700, 600
    a = np.random.default_rng(1).standard_normal((m, n))
    da = zb.colmajor_to_device(a)
    dq, dh = torch.zeros_like(da), torch.zeros((n, n), dtype=torch.float64, device="cuda")
    out = [(torch.zeros_like(da), torch.zeros_like(dh)) for _ in range(2)]

    def qdwh():
        return zb.lib().zolo_qdwh_dev(h.ptr, b"N", m, n, 0.0, da.data_ptr(), m, dq.data_ptr(), m, dh.data_ptr(), n, 0,
                                      12, 0)

    def batch():
        return zb.qdwh_batch_dev(h, [(m, n, da.data_ptr(), m, q.data_ptr(), m, hh.data_ptr(), n) for q, hh in out])

    assert qdwh() == 0
    q0 = dq.clone()
    batch()
    batch()  # its bucket as a captured graph
    h.set_option(zb.OPT_PANEL_WAIT, -1)
    assert qdwh() == WAIT_RAN_OUT
    with pytest.raises(zb.ZoloError) as e:
        batch()
    assert e.value.info == WAIT_RAN_OUT
    h.set_option(zb.OPT_PANEL_WAIT, 0)
    assert qdwh() == 0 and torch.equal(dq, q0)
    info, _ = batch()
    assert all(x == 0 for x in info)


def test_option_values(h):
    assert zb.lib().zolo_set_option(h.ptr, zb.OPT_PANEL_WAIT, -2) == -3
    h.set_option(zb.OPT_PANEL_WAIT, -1)
    assert h.get_option(zb.OPT_PANEL_WAIT) == -1


def test_code_is_not_left_for_the_next_call(h):
    """A call in which a wait ran out and which then ends with another error keeps its code to itself."""
    import torch
    m, n = 700, 64
    dx = zb.colmajor_to_device(np.random.default_rng(2).standard_normal((m, n)))
    dz = torch.zeros((n, m + 2), dtype=torch.float64, device="cuda")

    def zoloqr(ptr):
        return zb.lib().zolo_zoloqr_dev(h.ptr, m, n, dx.data_ptr(), m, 0.5, 1.0, ptr, m + 2)

    h.set_option(zb.OPT_PANEL_WAIT, -1)
    # Z off an 8-byte boundary: refused on the host (716) at the last product, after the panels
    assert zoloqr(dz.data_ptr() + 4) == -1716
    h.set_option(zb.OPT_PANEL_WAIT, 0)
    assert zoloqr(dz.data_ptr()) == 0
