"""TSQR / panel QR kernels (C ABI) vs the oracle restatement of panelQR/hou_tsqr_panel."""
import numpy as np
import pytest
import torch

from oracle import algos as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [32, 64, 96, 128, 160, 256, 544, 1024, 4128, 16352])
def test_tsqr_matches_oracle(cuda, evdlib, m):
    A = np.random.default_rng(m).standard_normal((m, 32))
    Qr, Rr = O.tsqr(A)
    Ad = evdlib.to_cm(torch.from_numpy(A), device=cuda)
    Q, R = evdlib.tsqr(Ad)
    torch.cuda.synchronize()
    Q, R = Q.cpu().numpy(), R.cpu().numpy()
    assert np.abs(R - Rr).max() <= 1e-12 * np.abs(Rr).max()
    assert np.abs(Q - Qr).max() <= 1e-12
    assert np.abs(Q.T @ Q - np.eye(32)).max() <= 1e-13
    assert np.abs(Q @ R - A).max() <= 1e-12 * np.abs(A).max()


@pytest.mark.parametrize("m", [32, 96, 128, 160, 640, 1056, 8192])
def test_panel_qr_matches_oracle(cuda, evdlib, m):
    A = np.random.default_rng(100 + m).standard_normal((m, 32))
    Yr, Wr, Rr = O.panel_qr(A)
    Ad = evdlib.to_cm(torch.from_numpy(A), device=cuda)
    Y, W, R = evdlib.panel_qr(Ad)
    torch.cuda.synchronize()
    Y, W, R = Y.cpu().numpy(), W.cpu().numpy(), R.cpu().numpy()
    assert np.abs(R - Rr).max() <= 1e-12 * np.abs(Rr).max()
    assert np.abs(Y - Yr).max() <= 1e-11
    assert np.abs(W - Wr).max() <= 1e-11
    # Householder form: unit lower Y, Q = I - W Y^T orthogonal, Q^T A = [R; 0]
    assert np.abs(np.triu(Y[:32], 1)).max() == 0.0
    assert np.abs(np.diag(Y[:32]) - 1.0).max() == 0.0
    Qf = np.eye(m) - W @ Y.T
    assert np.abs(Qf.T @ Qf - np.eye(m)).max() <= 1e-13 * 10
    QtA = Qf.T @ A
    assert np.abs(QtA[:32] - R).max() <= 1e-12 * np.abs(A).max() * 4
    if m > 32:
        assert np.abs(QtA[32:]).max() <= 1e-12 * np.abs(A).max() * 4


def test_panel_rejects_bad_shapes(cuda, evdlib):
    A = evdlib.to_cm(torch.randn(100, 32, dtype=torch.float64), device=cuda)  # m % 32 != 0
    with pytest.raises(evdlib.EvdError):
        evdlib.panel_qr(A)


@pytest.mark.parametrize("m", [256, 544, 4128])
def test_a_tree_wait_that_runs_out_is_reported_and_stays_visible(cuda, evdlib, m):
    """The first leaf never runs: its parent's wait ends with a status and NaN,
    and so does a panel on the counters that this leaves behind; a call that
    resets them is right again."""
    import ctypes as C
    A = torch.from_numpy(np.random.default_rng(m).standard_normal((m, 32)))
    work = torch.zeros(evdlib.lib().evd_panel_qr_work_size(m, 32), dtype=torch.float64,
                       device=cuda)
    for fresh in (1, 0):
        Ad = evdlib.to_cm(A, device=cuda)
        R = torch.zeros(32, 32, dtype=torch.float64, device=cuda)
        torch.cuda.synchronize()
        rc = evdlib.lib().evd_test_tsqr_timeout(
            C.c_long(m), C.c_void_p(Ad.data_ptr()), C.c_long(m), C.c_void_p(R.data_ptr()),
            C.c_void_p(work.data_ptr()), C.c_int(fresh), C.c_long(2000000), None)
        assert rc == -3  # EVD_ERR_TIMEOUT
        assert torch.isnan(torch.triu(R.t())).sum() == 32 * 33 // 2
    Ad, R = evdlib.to_cm(A, device=cuda), evdlib.empty_cm(32, 32, device=cuda)
    rc = evdlib.lib().evd_tsqr(m, 32, C.c_void_p(Ad.data_ptr()), m, C.c_void_p(R.data_ptr()), 32,
                               C.c_void_p(work.data_ptr()), work.numel(), None)
    torch.cuda.synchronize()
    assert rc == 0
    Rr = O.tsqr(A.numpy())[1]
    assert np.abs(R.cpu().numpy() - Rr).max() <= 1e-12 * np.abs(Rr).max()


def test_reciprocal_of_the_panel_lu(cuda, evdlib):
    """Two Newton steps from the hardware's approximation (2^-20 or better): the
    error left is the last rounding, so within one ulp of the division."""
    import ctypes as C
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(1.0, 2.0, 100000),  # the LU's pivots
                        rng.choice([-1.0, 1.0], 100000) * 10.0 ** rng.uniform(-290, 290, 100000),
                        2.0 ** np.arange(-960, 961), np.nextafter(2.0 ** np.arange(-960, 961), 0)])
    xd = torch.from_numpy(x).to(cuda)
    y = torch.empty_like(xd)
    torch.cuda.synchronize()
    assert evdlib.lib().evd_test_reciprocal(C.c_long(x.size), C.c_void_p(xd.data_ptr()),
                                            C.c_void_p(y.data_ptr()), None) == 0
    want = 1.0 / x
    assert (np.abs(y.cpu().numpy() - want) <= np.spacing(np.abs(want))).all()


def test_panel_and_band_reduction_in_a_stream_capture(cuda, evdlib):
    """Captured, the chains of kernels with programmatic launches and the tree's
    counters replay to the same bits."""
    n, nb = 512, 128
    A = evdlib.to_cm(torch.from_numpy(O.sym_gaussian(n, 5)), device=cuda)
    names = ("OA", "dA", "W", "Y")
    buf = {k: evdlib.zeros_cm(n, n, device=cuda) for k in names}
    Z, R = evdlib.zeros_cm(n, nb, device=cuda), evdlib.zeros_cm(n, nb, device=cuda)
    lw = evdlib.lib().evd_sy2sb_work_size(n, 32, nb)
    work = torch.zeros(lw, dtype=torch.float64, device=cuda)

    def reduce(stream):
        buf["OA"].copy_(A)
        buf["dA"].copy_(A)
        buf["W"].zero_()
        buf["Y"].zero_()
        args = []
        for t in (*(buf[k] for k in names), Z, R):
            args.extend(evdlib._cm(t, "x"))
        evdlib.call("evd_sy2sb", n, n, 32, nb, *args, evdlib._ptr(work), lw,
                    evdlib._stream(stream))

    reduce(None)
    torch.cuda.synchronize()
    want = [buf[k].clone() for k in ("dA", "W", "Y")]
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        reduce(s)
    for _ in range(3):
        for k in names:
            buf[k].fill_(7.0)
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(buf[k], w) for k, w in zip(("dA", "W", "Y"), want))
