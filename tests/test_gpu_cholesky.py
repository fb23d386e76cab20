"""Batched Cholesky on the device against the reference's outputs (tests/golden),
the C oracle (a restatement of linalg.cpp:117-136) and numpy.

Bar: per matrix, ||L - L_oracle|| <= 1e-12 * cond(A) * ||L_oracle|| (Frobenius),
the same normwise bound the solve path is held to; the upper triangle of A is
never read; a matrix that is not positive definite fails the call."""
import ctypes as C

import numpy as np
import pytest

from numpp_b200 import _lib
from numpp_b200 import linalg as la

pytestmark = pytest.mark.gpu


def _spd(seed, cnt, n):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((cnt, n, n))
    A = X @ X.transpose(0, 2, 1) / n + np.eye(n)
    A += np.triu(rng.standard_normal((cnt, n, n)), 1)  # the upper triangle must not matter
    return A


def _close(L, Lo, A):
    sym = np.tril(A) + np.tril(A, -1).transpose(0, 2, 1)
    cond = np.linalg.cond(sym)
    err = np.linalg.norm((L - Lo).reshape(len(L), -1), axis=1)
    return np.all(err <= 1e-12 * cond * np.linalg.norm(Lo.reshape(len(L), -1), axis=1))


def test_cholesky_golden(golden, lib):
    """test_linalg.cpp:61-69, test_batched_linalg.cpp:53-58 and a seeded stack."""
    A = golden["spd3_A"]
    np.testing.assert_allclose(la.cholesky(A), golden["chol_spd3"], rtol=1e-14, atol=1e-15)
    np.testing.assert_allclose(la.cholesky(golden["chol_stack_A"]), golden["chol_stack_L"], rtol=1e-14, atol=1e-15)
    L = la.cholesky(golden["chol40_A"])
    assert _close(L, golden["chol40_L"], golden["chol40_A"])
    with pytest.raises(la.LinAlgError, match=str(golden["chol_notpd_err"])):
        la.cholesky(np.array([[-1.0, 0], [0, -1]]))


@pytest.mark.parametrize("cnt,n", [(64, 1), (50, 5), (40, 16), (33, 32), (20, 33), (12, 100), (6, 300),
                                   (3, 513), (2, 1030)])
def test_cholesky_vs_oracle(oracle, lib, cnt, n):
    A = _spd(n, cnt, n)
    L = la.cholesky(A)
    Lo, ok = oracle.cholesky(A)
    assert ok.all()
    assert np.array_equal(L, np.tril(L))
    assert _close(L, Lo, A)
    sym = np.tril(A) + np.tril(A, -1).transpose(0, 2, 1)
    np.testing.assert_allclose(L @ L.transpose(0, 2, 1), sym, rtol=0, atol=1e-12 * np.abs(sym).max())


@pytest.mark.parametrize("n", [6, 40, 600])
def test_not_positive_definite(lib, n):
    A = _spd(7, 3, n)
    A[1, n // 2, n // 2] = -5.0  # system 1 fails at (or before) column n // 2
    with pytest.raises(la.LinAlgError, match="Matrix is not positive definite"):
        la.cholesky(A)
    Lm = np.empty_like(A)
    info = np.full(3, -1, np.int32)
    assert lib.nppb_cholesky_batched(3, n, _lib.ptr(A), _lib.ptr(Lm), _lib.ptr(info)) == _lib.OK
    assert info[0] == 0 and info[2] == 0 and 1 <= info[1] <= n // 2 + 1
    Lo, ok = __import__("oracle").load_oracle().cholesky(A[[0, 2]])
    assert _close(Lm[[0, 2]], Lo, A[[0, 2]])


def test_cholesky_device_entry(lib, oracle):
    import torch
    A = _spd(11, 4, 200)
    dA = torch.from_numpy(A).cuda()
    dL = torch.empty_like(dA)
    dI = torch.zeros(4, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    rc = lib.nppb_d_cholesky_batched(4, 200, C.c_void_p(dA.data_ptr()), C.c_void_p(dL.data_ptr()),
                                     C.c_void_p(dI.data_ptr()), C.c_void_p(st))
    assert rc == _lib.OK, _lib.last_error()
    torch.cuda.synchronize()
    assert not dI.any()
    Lo, _ = oracle.cholesky(A)
    assert _close(dL.cpu().numpy(), Lo, A)
    assert lib.nppb_d_cholesky_batched(1, 5000, None, None, None, None) == _lib.E_RANGE


@pytest.mark.parametrize("n", [1, 7, 33, 70, 300])
def test_roots_of_squares_and_of_infinity(lib, n):
    """The factor of a diagonal of squares is their roots, without rounding; an infinite entry's
    root is infinite and its column's multipliers are zero (linalg.cpp:126-133)."""
    A = np.zeros((8, n, n))
    roots = np.arange(1.0, 8 * n + 1).reshape(8, n)
    A[:, range(n), range(n)] = roots ** 2
    L = la.cholesky(A)
    np.testing.assert_array_equal(L[:, range(n), range(n)], roots)
    assert np.count_nonzero(L) == 8 * n
    if n > 1:
        A[0, 0, 0], A[0, n - 1, 0] = np.inf, 5.0
        L = la.cholesky(A[:1])[0]
        assert L[0, 0] == np.inf and L[n - 1, 0] == 0.0
        np.testing.assert_array_equal(L[range(1, n), range(1, n)], roots[0, 1:])


@pytest.mark.parametrize("n", [2048, 2049, 2050, 2176, 2300])
@pytest.mark.parametrize("inplace", [False, True])
def test_outer_blocks(lib, n, inplace):
    """Orders above 2048 go by outer blocks of 128 columns: odd and even ones, partial last blocks,
    matrices that are not positive definite in the first, a middle and the last block, with NaN
    above the diagonal. Bar: 8 (n + 2) eps cond(A) of the factor (test_gpu_resident.py)."""
    torch = pytest.importorskip("torch")
    P, st = _lib.ptr, torch.cuda.current_stream().cuda_stream
    bad = [None, 5, 1500, n - 1]
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    W = torch.randn(1, n, n, dtype=torch.float64, device="cuda", generator=g)
    A0 = W[0] @ W[0].T
    A0.diagonal().add_(float(n))
    A = A0.tril().repeat(4, 1, 1)
    A[:, torch.triu(torch.ones(n, n, device="cuda"), 1).bool()] = float("nan")
    for s, b in enumerate(bad):
        if b is not None:
            A[s, b, b] = -1.0
    L = A if inplace else torch.full_like(A, 7.0)
    info = torch.full((4,), -1, dtype=torch.int32, device="cuda")
    assert lib.nppb_d_cholesky_batched(4, n, P(A), P(L), P(info), st) == _lib.OK, _lib.last_error()
    assert info.tolist() == [0 if b is None else b + 1 for b in bad]
    want = np.linalg.cholesky(A0.cpu().numpy())
    got = L[0].cpu().numpy()
    assert not np.triu(got, 1).any()
    assert np.abs(got - want).max() <= 8 * (n + 2) * 2.0 ** -53 * np.linalg.cond(A0.cpu().numpy()) * np.abs(want).max()
