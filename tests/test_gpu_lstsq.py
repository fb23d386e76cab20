"""lstsq, svdvals and the 2-norm cond on the device against the reference's
outputs (tests/golden, from its Jacobi-SVD lstsq) and numpy.

Bars: singular values within 1e-13 * s_max; rank exact; the solution within
1e-12 * cond(A) relative to its norm (cond over the kept singular values);
residuals within 1e-10 relative (they are differences of nearly equal
quantities only when the fit is nearly exact, and then they are tiny)."""
import ctypes as C

import numpy as np
import pytest

from numpp_b200 import _lib
from numpp_b200 import linalg as la

pytestmark = pytest.mark.gpu

KEYS = ("R", "W", "tall", "wide", "sq", "def")


def _check(A, b, x, res, rk, sv, xo, reso, rko, svo):
    assert rk == rko
    np.testing.assert_allclose(sv, svo, rtol=0, atol=1e-13 * svo[0])
    kept = svo[svo > svo[0] * 2.220446049250313e-16 * max(A.shape)]
    cond = kept[0] / kept[-1]
    assert np.linalg.norm(x - xo) <= 1e-12 * cond * max(np.linalg.norm(xo), 1e-300)
    assert res.shape == reso.shape
    if reso.size:
        np.testing.assert_allclose(res, reso, rtol=1e-10, atol=1e-12 * np.abs(b).max() ** 2)


def test_lstsq_golden(golden, lib):
    for key in KEYS:
        A, b = golden[f"lsq_{key}_A"], golden[f"lsq_{key}_b"]
        x, res, rk, sv = la.lstsq(A, b)
        _check(A, b, x, res, rk, sv, golden[f"lsq_{key}_x"], golden[f"lsq_{key}_res"],
               int(golden[f"lsq_{key}_rank"]), golden[f"lsq_{key}_s"])


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (5, 3, 1), (3, 5, 2), (200, 64, 4), (64, 200, 3), (512, 32, 8),
                                   (3000, 8, 2), (40, 40, 5)])
def test_lstsq_vs_oracle(oracle, lib, m, n, k):
    rng = np.random.default_rng(m * 7 + n)
    A = rng.standard_normal((m, n))
    b = rng.standard_normal((m, k))
    x, res, rk, sv = la.lstsq(A, b)
    xo, reso, rko, svo = oracle.lstsq(A, b)
    _check(A, b, x, res, rk, sv, xo, reso, rko, svo)
    xn = np.linalg.lstsq(A, b, rcond=None)[0]
    np.testing.assert_allclose(x, xn, rtol=1e-9, atol=1e-10 * np.abs(xn).max())


def test_rank_deficient_minimum_norm(lib, oracle):
    rng = np.random.default_rng(3)
    A = rng.standard_normal((30, 5)) @ rng.standard_normal((5, 12))  # rank 5
    b = rng.standard_normal(30)
    x, res, rk, sv = la.lstsq(A, b)
    xo, reso, rko, svo = oracle.lstsq(A, b)
    assert rk == rko == 5 and res.size == 0
    np.testing.assert_allclose(x, np.linalg.pinv(A) @ b, rtol=1e-8, atol=1e-10)
    np.testing.assert_allclose(x, xo, rtol=1e-8, atol=1e-10)


def test_svdvals_and_cond(lib):
    rng = np.random.default_rng(4)
    A = rng.standard_normal((6, 2, 50, 30))
    np.testing.assert_allclose(la.svdvals(A), np.linalg.svd(A, compute_uv=False), rtol=1e-12, atol=1e-13)
    S = rng.standard_normal((4, 20, 20)) + 3 * np.eye(20)
    for p in (None, 2, -2):
        np.testing.assert_allclose(la.cond(S, p), np.linalg.cond(S, p), rtol=1e-11)
    assert la.cond(np.zeros((3, 3))) == np.inf and la.cond(np.zeros((3, 3)), -2) == 0.0


def test_declined_and_device_entry(lib):
    import torch
    with pytest.raises(la.Declined):
        la.lstsq(np.ones((100, 100)), np.ones(100))      # min(m, n) = 100 > 64
    rng = np.random.default_rng(5)
    A = rng.standard_normal((7, 40, 10))
    B = rng.standard_normal((7, 40, 2))
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    dX = torch.empty(7, 10, 2, dtype=torch.float64, device="cuda")
    dS = torch.empty(7, 10, dtype=torch.float64, device="cuda")
    dR = torch.empty(7, dtype=torch.int32, device="cuda")
    dres = torch.empty(7, 2, dtype=torch.float64, device="cuda")
    dh = torch.empty(7, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    rc = lib.nppb_d_lstsq_batched(7, 40, 10, 2, C.c_void_p(dA.data_ptr()), C.c_void_p(dB.data_ptr()), -1.0,
                                  C.c_void_p(dX.data_ptr()), C.c_void_p(dS.data_ptr()), C.c_void_p(dR.data_ptr()),
                                  C.c_void_p(dres.data_ptr()), C.c_void_p(dh.data_ptr()), C.c_void_p(st))
    assert rc == _lib.OK, _lib.last_error()
    torch.cuda.synchronize()
    assert bool((dR == 10).all()) and bool((dh == 1).all())
    for i in range(7):
        xn, rn = np.linalg.lstsq(A[i], B[i], rcond=None)[:2]
        np.testing.assert_allclose(dX[i].cpu().numpy(), xn, rtol=1e-10, atol=1e-12)
        np.testing.assert_allclose(dres[i].cpu().numpy(), rn, rtol=1e-10)


def test_rcond_and_wide_rank_deficient(lib, oracle):
    """An explicit rcond drops the same singular values as the reference; a
    wide rank-deficient problem gives the minimum-norm solution."""
    rng = np.random.default_rng(8)
    A = rng.standard_normal((25, 12)) @ np.diag(np.logspace(0, -9, 12)) @ rng.standard_normal((12, 12))
    b = rng.standard_normal((25, 2))
    for rcond in (1e-4, 1e-7, 0.0):
        x, res, rk, sv = la.lstsq(A, b, rcond=rcond)
        xo, reso, rko, svo = oracle.lstsq(A, b, rcond)
        assert rk == rko, rcond
        np.testing.assert_allclose(sv, svo, rtol=0, atol=1e-13 * svo[0])
        if rk < 12:
            np.testing.assert_allclose(x, xo, rtol=1e-8, atol=1e-9 * np.abs(xo).max())
    W = rng.standard_normal((6, 3)) @ rng.standard_normal((3, 20))  # 6 x 20, rank 3
    bw = rng.standard_normal(6)
    x, res, rk, sv = la.lstsq(W, bw)
    assert rk == 3 and res.size == 0
    np.testing.assert_allclose(x, np.linalg.pinv(W) @ bw, rtol=1e-8, atol=1e-10)


@pytest.mark.parametrize("m,n,k", [
    (63, 31, 1), (64, 31, 1), (64, 32, 9), (65, 33, 2), (127, 63, 1), (128, 64, 20),  # both sides of the reduction's rule
    (64, 1, 2), (65, 2, 8), (200, 3, 17), (20, 130, 11), (31, 63, 1), (1, 100, 3), (340, 64, 16), (23, 24, 5)])
def test_reduced_and_direct_sweeps(lib, m, n, k):
    """Problems at the edges of the reduction to the triangle (max >= 2 min, max >= 64), odd and
    even column counts, right-hand sides in one group and in several, against numpy's SVD: a
    backward-stable solution is within a few (m + n) eps cond of it, singular values within a few
    (m + n) eps of s_max."""
    rng = np.random.default_rng(m * 131 + n * 7 + k)
    A = rng.standard_normal((3, m, n))
    B = rng.standard_normal((3, m, k))
    X, S, resid = np.zeros((3, n, k)), np.zeros((3, min(m, n))), np.zeros((3, k))
    rank, has = np.zeros(3, np.int32), np.zeros(3, np.int32)
    P = _lib.ptr
    rc = lib.nppb_lstsq_batched(3, m, n, k, P(A), P(B), -1.0, P(X), P(S), P(rank), P(resid), P(has))
    assert rc == _lib.OK, _lib.last_error()
    eps = np.finfo(float).eps
    for i in range(3):
        s = np.linalg.svd(A[i], compute_uv=False)
        x = np.linalg.pinv(A[i]) @ B[i]
        cond = s[0] / s[-1]
        np.testing.assert_allclose(S[i], s, rtol=0, atol=20 * (m + n) * eps * s[0])
        assert rank[i] == min(m, n) and has[i] == (m > n)
        assert np.linalg.norm(X[i] - x) <= 50 * (m + n) * eps * cond ** 2 * max(np.linalg.norm(x), 1.0)
        if m > n:
            r = ((A[i] @ x - B[i]) ** 2).sum(axis=0)
            np.testing.assert_allclose(resid[i], r, rtol=0, atol=100 * (m + n) * eps * (B[i] ** 2).sum(axis=0).max())


def test_nan_and_infinity_stay_where_they_are(lib):
    """A NaN (or an infinity) in one column is that column's singular value; the other values are
    those of the matrix without it, in tall problems (reduced to the triangle when finite) too."""
    rng = np.random.default_rng(11)
    for bad in (np.nan, np.inf):
        for col in (0, 4, 9):
            A, b = rng.standard_normal((100, 10)), rng.standard_normal(100)
            A[17, col] = bad
            sv = la.lstsq(A, b)[3]
            assert np.count_nonzero(np.isfinite(sv)) == 9
            np.testing.assert_allclose(np.sort(sv[np.isfinite(sv)])[::-1],
                                       np.linalg.svd(np.delete(A, col, 1), compute_uv=False), rtol=1e-12)


@pytest.mark.parametrize("shift", [60, 100, 126, 140, 153, 300, 480])
@pytest.mark.parametrize("m,n,col", [(40, 6, 0), (40, 6, 5), (100, 33, 16)])
def test_columns_of_very_different_lengths(lib, m, n, col, shift):
    """Scaling a column by a power of two scales its unknown by the inverse and changes nothing
    else, also where the pair's rotation angle is far below FP32's range (rcond = 0: every column
    counts). Bar: that of the unscaled problem (test_reduced_and_direct_sweeps)."""
    rng = np.random.default_rng(m + col)
    A, b = rng.standard_normal((m, n)), rng.standard_normal(m)
    x0 = np.linalg.lstsq(A, b, rcond=None)[0]
    s = np.linalg.svd(A, compute_uv=False)
    As = A.copy()
    As[:, col] *= 2.0 ** -shift
    x, _, rank, _ = la.lstsq(As, b, rcond=0.0)
    assert rank == n
    x[col] *= 2.0 ** -shift
    eps = np.finfo(float).eps
    assert np.linalg.norm(x - x0) <= 50 * (m + n) * eps * (s[0] / s[-1]) ** 2 * np.linalg.norm(x0)


@pytest.mark.parametrize("m,n,k", [(200, 32, 1), (200, 32, 11), (64, 32, 3), (20, 90, 2)])
@pytest.mark.parametrize("shift", [-600, -518, -505, -300, 300, 478, 500, 505])
def test_entries_towards_the_ends_of_the_range(lib, m, n, k, shift):
    """A scaled by a power of two scales S and the inverse of X; nothing else changes. Squares of
    2^-518 are subnormal: their sums hold 2^-1074 / 2^(-1036 + 7) of a norm, and S with them;
    those of 2^-600 are zero, and so is every singular value."""
    rng = np.random.default_rng(m + k)
    A, B = rng.standard_normal((m, n)), rng.standard_normal((m, k))
    x, res, rank, s = la.lstsq(np.ldexp(A, shift), B)
    if shift == -600:
        assert rank == 0 and not s.any() and not x.any()
        return
    s0 = np.linalg.svd(A, compute_uv=False)
    x0 = np.linalg.pinv(A) @ B
    assert rank == min(m, n)
    rel = 1e-9 if shift == -518 else 50 * (m + n) * np.finfo(float).eps * (s0[0] / s0[-1]) ** 2
    np.testing.assert_allclose(np.ldexp(s, -shift), s0, rtol=rel)
    assert np.linalg.norm(np.ldexp(x, shift) - x0) <= rel * np.linalg.norm(x0)
    if m > n:
        np.testing.assert_allclose(res, ((A @ x0 - B) ** 2).sum(axis=0), rtol=1e-8)


@pytest.mark.parametrize("col", [0, 7, 31])
@pytest.mark.parametrize("shift", [-600, -518, -480, -200, 200, 500])
def test_one_column_towards_the_ends_of_the_range(lib, col, shift):
    """Default tolerance: a tiny column counts as none, beside a huge one the others do."""
    rng = np.random.default_rng(col)
    A, B = rng.standard_normal((200, 32)), rng.standard_normal((200, 2))
    A[:, col] = np.ldexp(A[:, col], shift)
    x, _, rank, s = la.lstsq(A, B)
    keep = np.arange(32) != col if shift < 0 else np.arange(32) == col
    want = np.zeros((32, 2))
    want[keep] = np.linalg.lstsq(A[:, keep], B, rcond=None)[0]
    assert rank == keep.sum() and np.isfinite(s).all()
    assert np.linalg.norm(x[keep] - want[keep]) <= 1e-10 * np.linalg.norm(want[keep])


@pytest.mark.parametrize("j", [0, 9])
@pytest.mark.parametrize("value", [np.nan, np.inf, 2.0 ** 1000])
def test_right_hand_sides_out_of_range_stay_alone(lib, j, value):
    rng = np.random.default_rng(5)
    A, B = rng.standard_normal((100, 20)), rng.standard_normal((100, 12))
    C = B.copy()
    C[3, j] = value
    x0 = la.lstsq(A, B)[0]
    x = la.lstsq(A, C)[0]
    others = np.arange(12) != j
    np.testing.assert_allclose(x[:, others], x0[:, others], rtol=1e-10, atol=1e-12)
    if np.isfinite(value):
        np.testing.assert_allclose(x[:, j], np.linalg.pinv(A)[:, 3] * value, rtol=1e-10)
