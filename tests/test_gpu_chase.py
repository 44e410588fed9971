"""Bulge chasing kernel (C ABI) vs the oracle restatement of the reference kernel."""
import numpy as np
import pytest
import torch
from scipy.linalg import eigvalsh_tridiagonal

from oracle import algos as O

pytestmark = pytest.mark.gpu


def _banded(n, b, seed):
    A = O.sym_gaussian(n, seed)
    return np.tril(np.triu(A, -b), b)


@pytest.mark.parametrize("n", [3, 4, 5, 33, 34, 64, 65, 100, 257, 512])
def test_chase_matches_oracle(cuda, evdlib, n):
    b = 32
    B = _banded(n, b, seed=n)
    sub_ref = O.band_pack(B, b)
    d_ref, e_ref, U_ref, _ = O.bulge_chase(sub_ref, n, b)

    Bd = evdlib.to_cm(torch.from_numpy(B), device=cuda)
    sub = evdlib.band_pack(Bd, b)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(sub.cpu().numpy(), sub_ref)  # exact copy kernel

    d, e, U = evdlib.bulge_chase(sub, b)
    torch.cuda.synchronize()
    scale = np.abs(B).max()
    assert np.abs(d.cpu().numpy() - d_ref).max() <= 1e-12 * scale * n
    assert np.abs(e.cpu().numpy() - e_ref).max() <= 1e-12 * scale * n
    assert np.abs(U.cpu().numpy() - U_ref).max() <= 1e-10
    # invariants: same spectrum, reflectors reproduce T
    if n > 1:
        w_t = eigvalsh_tridiagonal(d.cpu().numpy(), e.cpu().numpy())
        w_b = np.linalg.eigvalsh(B)
        assert np.abs(w_t - w_b).max() <= 1e-12 * np.linalg.norm(B, 2) * 8
        Un = U.cpu().numpy()
        Q2 = O.q2_apply(np.eye(n), Un, n, b, transpose=False)
        T = np.diag(d.cpu().numpy()) + np.diag(e.cpu().numpy(), 1) + np.diag(e.cpu().numpy(), -1)
        assert np.abs(Q2.T @ B @ Q2 - T).max() <= 1e-13 * np.linalg.norm(B, 2) * 8


@pytest.mark.parametrize("n", [2048, 4100])
def test_chase_spectrum_large(cuda, evdlib, n):
    b = 32
    B = _banded(n, b, seed=7)
    Bd = evdlib.to_cm(torch.from_numpy(B), device=cuda)
    sub = evdlib.band_pack(Bd, b)
    d, e, U = evdlib.bulge_chase(sub, b)
    torch.cuda.synchronize()
    w_t = eigvalsh_tridiagonal(d.cpu().numpy(), e.cpu().numpy())
    w_b = np.linalg.eigvalsh(B)
    assert np.abs(w_t - w_b).max() <= 1e-12 * np.linalg.norm(B, 2) * 8
    # reflector norms: ||u||^2 = 2 for every stored reflector segment
    Un = U.cpu().numpy()
    seg = Un[1:33, 0]
    assert abs(seg @ seg - 2.0) < 1e-12


def test_chase_repeatable(cuda, evdlib):
    """Two calls in one process give identical results (the reference's
    g_overFlag made a second call return immediately)."""
    n, b = 300, 32
    B = _banded(n, b, seed=3)
    Bd = evdlib.to_cm(torch.from_numpy(B), device=cuda)
    out = []
    for _ in range(2):
        sub = evdlib.band_pack(Bd, b)
        d, e, U = evdlib.bulge_chase(sub, b)
        out.append((d.clone(), e.clone(), U.clone()))
    torch.cuda.synchronize()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][2], out[1][2])


@pytest.mark.parametrize("n", [130, 131, 259, 515, 1027, 2050, 2051, 18950])
def test_chase_is_an_orthogonal_similarity(cuda, evdlib, n):
    """B Q2 Z = Q2 T Z on a few random vectors, at the orders where the chase
    changes its form (one CTA, clusters of 2 to 16, cooperative launches)."""
    b = 32
    g = torch.Generator(device=cuda).manual_seed(n)
    sub = torch.zeros(n, 2 * b, dtype=torch.float64, device=cuda)
    for o in range(b + 1):
        sub[: n - o, o] = torch.randn(n - o, generator=g, dtype=torch.float64, device=cuda)
    band = sub.clone()
    d, e, U = evdlib.bulge_chase(sub.t(), b)
    Z = evdlib.to_cm(torch.randn(n, 4, generator=g, dtype=torch.float64, device=cuda), device=cuda)
    TZ = d[:, None] * Z
    TZ[1:] += e[:, None] * Z[:-1]
    TZ[:-1] += e[:, None] * Z[1:]
    QTZ = evdlib.bc_back_apply(evdlib.to_cm(TZ, device=cuda), U)
    QZ = evdlib.bc_back_apply(Z.clone(memory_format=torch.preserve_format), U)
    BQZ = band[:, :1] * QZ
    for o in range(1, b + 1):
        BQZ[o:] += band[: n - o, o: o + 1] * QZ[: n - o]
        BQZ[: n - o] += band[: n - o, o: o + 1] * QZ[o:]
    # backward stable: a few units of rounding per reflector that a row meets
    norm2 = 2.0 * 65 ** 0.5  # of a random band matrix, from above to within a factor of 2
    assert (BQZ - QTZ).norm() <= 8e-13 * norm2 * Z.norm()


def _chase(evdlib, cuda, band, form, before=None):
    import ctypes as C
    n = band.shape[0]
    sub, U = band.clone(), torch.zeros(n, n, dtype=torch.float64, device=cuda)
    d = torch.empty(n, dtype=torch.float64, device=cuda)
    e = torch.empty(n, dtype=torch.float64, device=cuda)
    iw = torch.empty(evdlib.lib().evd_bulge_chase_iwork_size(n) // 4, dtype=torch.int32,
                     device=cuda)
    torch.cuda.synchronize()
    rc = evdlib.lib().evd_test_bulge_chase(
        C.c_long(n), C.c_void_p(sub.data_ptr()), C.c_void_p(U.data_ptr()), C.c_long(n),
        C.c_void_p(d.data_ptr()), C.c_void_p(e.data_ptr()), C.c_void_p(iw.data_ptr()),
        C.c_void_p(before.data_ptr() if before is not None else None), form, None)
    torch.cuda.synchronize()
    return rc, d, e[: n - 1], U


@pytest.mark.parametrize("n", [3, 34, 65, 100, 257, 512, 1100, 2200, 4200])
def test_ticketed_chase_agrees_with_the_pipeline(cuda, evdlib, n):
    """The kernel of orders beyond the pipeline, at orders that reach both."""
    g = torch.Generator(device=cuda).manual_seed(n)
    band = torch.zeros(n, 64, dtype=torch.float64, device=cuda)
    for o in range(min(33, n)):
        band[: n - o, o] = torch.randn(n - o, generator=g, dtype=torch.float64, device=cuda)
    rc, d, e, U = _chase(evdlib, cuda, band, 0)
    rt, dt, et, Ut = _chase(evdlib, cuda, band, 1)
    assert rc == 0 and rt == 0
    B = np.zeros((n, n))
    for o in range(min(33, n)):
        v = band[: n - o, o].cpu().numpy()
        B += np.diag(v, -o) + (np.diag(v, o) if o else 0)
    w = np.linalg.eigvalsh(B)
    for a, b in ((d, e), (dt, et)):
        wt = eigvalsh_tridiagonal(a.cpu().numpy(), b.cpu().numpy())
        assert np.abs(wt - w).max() <= 8e-12 * np.abs(w).max()
    # the first sweeps, where rounding has not grown yet, reflector by reflector
    assert (U[: min(n, 64), :8] - Ut[: min(n, 64), :8]).abs().max() <= 1e-10


def test_chase_reports_an_error_of_the_stages_before_it(cuda, evdlib):
    band = torch.zeros(100, 64, dtype=torch.float64, device=cuda)
    band[:, 0] = 1.0
    word = torch.tensor([2], dtype=torch.int32, device=cuda)
    assert _chase(evdlib, cuda, band, 0, word)[0] == -3  # EVD_ERR_TIMEOUT
    word.zero_()
    assert _chase(evdlib, cuda, band, 0, word)[0] == 0


@pytest.mark.parametrize("n", [2200, 4200])
def test_chase_whose_gate_shuts_is_done_by_the_ticketed_kernel(cuda, evdlib, n):
    g = torch.Generator(device=cuda).manual_seed(n)
    band = torch.zeros(n, 64, dtype=torch.float64, device=cuda)
    for o in range(33):
        band[: n - o, o] = torch.randn(n - o, generator=g, dtype=torch.float64, device=cuda)
    want = _chase(evdlib, cuda, band, 1)
    got = _chase(evdlib, cuda, band, 2)
    assert want[0] == 0 and got[0] == 0
    assert all(torch.equal(a, b) for a, b in zip(want[1:], got[1:]))


def test_cooperative_chases_on_streams_at_once(cuda, evdlib):
    """Together they ask for more SMs than there are; results as alone."""
    import threading
    orders = (12000, 9000, 2500, 11000, 4100, 10000)
    bands, want = [], []
    for n in orders:
        g = torch.Generator(device=cuda).manual_seed(n)
        band = torch.zeros(n, 64, dtype=torch.float64, device=cuda)
        for o in range(33):
            band[: n - o, o] = torch.randn(n - o, generator=g, dtype=torch.float64, device=cuda)
        bands.append(band)
        want.append(evdlib.bulge_chase(band.clone().t(), 32)[:2])
    torch.cuda.synchronize()
    got = [None] * len(orders)

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            sub = bands[i].clone()
            got[i] = evdlib.bulge_chase(sub.t(), 32, stream=s)[:2]
            s.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(orders))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    torch.cuda.synchronize()
    for band, a, b in zip(bands, want, got):
        if not torch.equal(a[0], b[0]):  # a gate that shut: the ticketed kernel's bits
            a = _chase(evdlib, cuda, band, 1)[1:3]
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
