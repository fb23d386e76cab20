"""The kernels that keep one system on a CTA, a cluster or a warp, at the edges
of their tiles and of the rules that choose them: blocks of 32 rows, one CTA up
to order 512, outer blocks of 128 columns above, strips of 32 right-hand sides,
clusters for few systems; and the tiles of the stacked product and of the
refinement residual.

The bar: LU with partial pivoting is backward stable, so a solution is within
n eps times a modest growth factor of the true one per unit of cond(A); with
n <= 1100 and growth 8 that is 1e-12 cond(A), which the other parity tests use
too. A product's entries are within (k + 2) eps sum |a||b|. Solutions of signed
permutation matrices, where no rounding occurs, are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def torch(lib):
    import torch
    return torch


def close(got, want, A, what):
    """max |got - want| <= 1e-12 cond(A) max |want|, system by system."""
    for s in range(len(A)):
        bound = 1e-12 * np.linalg.cond(A[s]) * np.abs(want[s]).max()
        err = np.abs(got[s] - want[s]).max()
        assert err <= bound, (what, s, err, bound)


def draw(seed, count, n, k):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((count, n, n)), rng.standard_normal((count, n, k))


@pytest.mark.parametrize("n", [1, 2, 8, 9, 31, 32, 33, 63, 64, 65, 95, 97, 255, 256, 257, 511, 512, 513, 639, 641, 1025])
@pytest.mark.parametrize("k", [1, 9, 33])
def test_solve_inverse_slogdet_at_the_edges(torch, n, k):
    from numpp_b200 import device
    A, B = draw(n * 100 + k, 3, n, k)
    dA = torch.from_numpy(A).cuda()
    X, info = device.solve(dA, torch.from_numpy(B).cuda(), check=False)
    assert not info.any()
    close(X.cpu().numpy(), np.linalg.solve(A, B), A, "solve")
    if k == 9:
        close(device.inv(dA).cpu().numpy(), np.linalg.inv(A), A, "inv")
        sign, logabs = device.slogdet(dA)
        rs, rl = np.linalg.slogdet(A)
        np.testing.assert_array_equal(sign.cpu().numpy(), rs)
        np.testing.assert_allclose(logabs.cpu().numpy(), rl, rtol=0, atol=1e-12 * max(np.linalg.cond(a) for a in A))


@pytest.mark.parametrize("n", [5, 32, 33, 70, 128, 200, 512, 513, 700])
def test_signed_permutations_are_exact_and_singular_systems_stop_alone(torch, n):
    """Every column has one candidate; a batch also holds a matrix with two equal
    columns of zeros, which stops with the column's number and leaves the others alone."""
    from numpp_b200 import device
    rng = np.random.default_rng(n)
    A = np.zeros((4, n, n))
    for s in range(4):
        A[s, rng.permutation(n), np.arange(n)] = rng.choice([-2.0, 0.5, 1.0], n)
    z = int(rng.integers(0, n))
    A[2, :, z] = 0.0
    B = rng.standard_normal((4, n, 3))
    X, info = device.solve(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), check=False)
    assert info.cpu().tolist() == [0, 0, z + 1, 0]
    for s in (0, 1, 3):
        want = np.empty_like(B[s])
        for j in range(n):
            i = int(np.nonzero(A[s, :, j])[0][0])
            want[j] = B[s, i] / A[s, i, j]
        np.testing.assert_array_equal(X[s].cpu().numpy(), want)


@pytest.mark.parametrize("n", [8, 32, 48, 64, 130])
def test_pivots_of_ties_and_of_equal_high_words(torch, n):
    """The first largest |a| in position order is taken, also where candidates
    differ only in the low half of their bits, or not at all."""
    from scipy.linalg import lu_factor
    from numpp_b200 import _lib
    rng = np.random.default_rng(n)
    A = np.stack([1.0 + rng.integers(0, 4, (n, n)) * 2.0 ** -40 + np.eye(n) * 0.25,
                  rng.choice([-1.0, 1.0], (n, n)) + np.diag(np.arange(n) * 2.0 ** -30)])
    dA = torch.from_numpy(A).cuda()
    LU = torch.empty_like(dA)
    piv, info = (torch.zeros(s, dtype=torch.int32, device="cuda") for s in ((2, n), (2,)))
    P = _lib.ptr
    rc = _lib.load().nppb_d_linalg_batched(2, n, 0, _lib.WANT_LU, P(dA), None, None, None, None, None, None, P(LU),
                                           P(piv), P(info), torch.cuda.current_stream().cuda_stream)
    assert rc == _lib.OK and not info.any()
    # the first column's pivot is decided before any rounding
    for s in range(2):
        assert int(piv[s, 0]) == int(np.argmax(np.abs(A[s, :, 0]))) == lu_factor(A[s])[1][0]


@pytest.mark.parametrize("n", [7, 33, 64, 512, 513, 777])
@pytest.mark.parametrize("count,k", [(2, 1), (2, 40), (160, 5)])
def test_kept_factors(torch, n, count, k):
    from numpp_b200 import _lib
    if count * n * n > 5e7:
        count = 20
    A, B = draw(n + k, count, n, k)
    A += np.sqrt(n) * np.eye(n)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    LU, X = torch.empty_like(dA), torch.empty_like(dB)
    piv, info = (torch.zeros(s, dtype=torch.int32, device="cuda") for s in ((count, n), (count,)))
    P, st = _lib.ptr, torch.cuda.current_stream().cuda_stream
    L = _lib.load()
    assert L.nppb_d_linalg_batched(count, n, 0, _lib.WANT_LU, P(dA), None, None, None, None, None, None, P(LU), P(piv),
                                   P(info), st) == _lib.OK
    assert L.nppb_d_getrs_batched(count, n, k, P(LU), P(piv), P(dB), P(X), st) == _lib.OK
    some = list(range(min(count, 4)))
    close(X.cpu().numpy()[some], np.linalg.solve(A[some], B[some]), A[some], "getrs")
    torch.testing.assert_close(dA @ X, dB, rtol=0, atol=1e-12 * n * float(X.abs().max()) * 2)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 65, 129, 257, 511, 513, 1025])
def test_cholesky_edges(torch, n):
    """In place, with NaN above the diagonal (never read), beside a matrix that is not positive definite."""
    from numpp_b200 import device
    rng = np.random.default_rng(n)
    G = rng.standard_normal((3, n, n))
    A = G @ G.transpose(0, 2, 1) + n * np.eye(n)
    bad = n // 2
    A[1, bad, bad] = -1.0
    H = A.copy()
    H[:, np.triu_indices(n, 1)[0], np.triu_indices(n, 1)[1]] = np.nan
    L, info = device.cholesky(torch.from_numpy(H).cuda(), check=False)
    assert info.cpu().tolist() == [0, bad + 1, 0]
    for s in (0, 2):
        want = np.linalg.cholesky(A[s])
        got = L[s].cpu().numpy()
        assert np.abs(got - want).max() <= 8 * (n + 2) * EPS * np.linalg.cond(A[s]) * np.abs(want).max()
        assert not np.triu(got, 1).any()


@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (32, 8, 32), (128, 16, 64), (129, 17, 65), (127, 33, 63), (31, 15, 130),
                                   (260, 2, 66), (96, 64, 96), (64, 47, 2)])
@pytest.mark.parametrize("shift", [0, 1])
def test_stacked_product(torch, m, k, n, shift):
    """shift = 1: operands on an odd 8-byte boundary (no 16-byte copies)."""
    from numpp_b200 import _lib
    rng = np.random.default_rng(m + k + n)
    A, B = rng.standard_normal((5, m, k)), rng.standard_normal((5, k, n))
    def put(a):
        t = torch.empty(a.size + shift, dtype=torch.float64, device="cuda")[shift:].view(a.shape)
        return t.copy_(torch.from_numpy(a))
    dA, dB, dC = put(A), put(B), put(np.full((5, m, n), np.nan))
    P = _lib.ptr
    assert _lib.load().nppb_d_gemm_batched(5, m, n, k, P(dA), P(dB), P(dC),
                                           torch.cuda.current_stream().cuda_stream) == _lib.OK
    err = np.abs(dC.cpu().numpy() - A @ B)
    assert (err <= 2 * (k + 2) * EPS * (np.abs(A) @ np.abs(B))).all()


@pytest.mark.parametrize("n", [33, 127, 128, 129, 385, 511, 1000])
@pytest.mark.parametrize("count,k", [(1, 1), (1, 8), (3, 3), (160, 2), (30, 11)])
def test_mixed_refinement_edges(torch, n, count, k):
    """Substitution chunks of 1 to 8 right-hand sides on clusters of 1 to 8 CTAs, the
    residual with fewer than, exactly and more than 8 of them, odd orders."""
    from numpp_b200 import _lib
    count = min(count, 80) if n > 400 else count
    A, B = draw(n + 7 * k, count, n, k)
    A += 2 * np.sqrt(n) * np.eye(n)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    X = torch.empty_like(dB)
    berr = torch.full((count,), np.nan, dtype=torch.float64, device="cuda")
    iters, fallback, info = (torch.full((count,), -1, dtype=torch.int32, device="cuda") for _ in range(3))
    P = _lib.ptr
    assert _lib.load().nppb_d_solve_mixed_batched(count, n, k, P(dA), P(dB), P(X), None, 1e-14, 30, 0, P(info), P(berr),
                                                  None, P(iters), P(fallback),
                                                  torch.cuda.current_stream().cuda_stream) == _lib.OK
    assert not info.any() and not fallback.any() and bool((iters >= 1).all()) and bool((berr <= 1e-14).all())
    some = list(range(min(count, 4)))
    close(X.cpu().numpy()[some], np.linalg.solve(A[some], B[some]), A[some], "mixed")
