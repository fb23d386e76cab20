"""The pivot search of the resident kernels (a CTA up to order 512, clusters above)
where the candidates' high words do not decide: ties across lanes, warps and CTAs,
candidates that differ in the low word only, subnormals.

Totally unimodular matrices (consecutive ones in every column) keep entries of 0
and +-1 through the whole elimination, so every column is a tie and every result
is exact: solutions, inverses and determinants are compared bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
ORDERS = [33, 64, 130, 257, 512, 513, 700, 1025]


@pytest.fixture(scope="module")
def torch(lib):
    import torch
    return torch


def unimodular(rng, n):
    A = np.zeros((n, n))
    for j in range(n):
        A[j:rng.integers(j, n) + 1, j] = 1.0
    A = A[rng.permutation(n)][:, rng.permutation(n)]
    return A * rng.choice([-1.0, 1.0], (n, 1)) * rng.choice([-1.0, 1.0], n)


@pytest.mark.parametrize("n", ORDERS)
@pytest.mark.parametrize("count", [1, 3, 40])
def test_every_column_a_tie(torch, n, count):
    from numpp_b200 import device
    if count * n > 20000:
        count = 20
    rng = np.random.default_rng(n + count)
    A = np.stack([unimodular(rng, n) for _ in range(min(count, 3))])
    A = A[np.arange(count) % len(A)]
    x = rng.integers(-9, 10, (count, n, 3)).astype(float)
    dA = torch.from_numpy(A).cuda()
    X, info = device.solve(dA, torch.from_numpy(A @ x).cuda(), check=False)
    assert not info.any()
    np.testing.assert_array_equal(X.cpu().numpy(), x)
    sign, logabs = device.slogdet(dA)
    np.testing.assert_array_equal(sign.cpu().numpy(), [round(np.linalg.slogdet(a)[0]) for a in A])
    assert not logabs.any()
    if count <= 3:
        inv = device.inv(dA).cpu().numpy()
        np.testing.assert_array_equal(A @ inv, np.broadcast_to(np.eye(n), A.shape))


@pytest.mark.parametrize("n", ORDERS)
def test_equal_high_words(torch, n):
    """The largest is found by its low word: multipliers stay at most 1, and with them the
    backward error within 8 n eps (test_gpu_backward.py). A first column of 1, 1 + 2^-40, ...
    shows the choice: its largest entry is the determinant's first factor."""
    from numpp_b200 import device
    rng = np.random.default_rng(n)
    A = 1.0 + rng.integers(0, 4096, (2, n, n)) * 2.0 ** -44 + np.eye(n) * 2.0 ** -30
    b = rng.standard_normal((2, n, 1))
    X, info = device.solve(torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda(), check=False)
    assert not info.any()
    X = X.cpu().numpy()
    for a, x, c in zip(A, X, b):
        r = np.abs(a.astype(np.longdouble) @ x.astype(np.longdouble) - c).max()
        assert r <= 8 * n * EPS * (np.abs(a).sum(axis=1).max() * np.abs(x).max() + np.abs(c).max())
    # one row decides: without the largest of column 0 as pivot the next column cancels to zero
    C = np.eye(n)
    C[:, 0] = 1.0 + rng.permutation(n) * 2.0 ** -50
    sign, logabs = device.slogdet(torch.from_numpy(np.stack([C, C])).cuda())
    rs, rl = np.linalg.slogdet(C)
    assert (sign.cpu().numpy() == rs).all() and np.abs(logabs.cpu().numpy() - rl).max() <= 4 * n * EPS


@pytest.mark.parametrize("n", [33, 130, 512, 513, 700])
def test_as_the_kept_factors_decide(torch, n):
    """Subnormals, zeros, infinities and NaN among the candidates: the same systems are
    singular, at the same column, as in the factorisation that keeps its factors, and the
    same determinants are numbers."""
    from numpp_b200 import _lib
    rng = np.random.default_rng(n)
    A = rng.standard_normal((12, n, n))
    c = int(rng.integers(1, n - 1))
    A[0, :, c] *= 2.0 ** -1060                       # a column of subnormals
    A[1, :, c] = 0.0
    A[2, :, c] = 0.0
    A[2, int(rng.integers(n)), c] = 2.0 ** -1074     # one candidate, the smallest number
    A[3, :, n - 1] *= 2.0 ** -1060
    A[4, :, c] = np.nan
    A[5, 5, c] = np.nan
    A[6, 7, 0] = np.nan
    A[7, 9, c] = np.inf
    A[8, :, c] = np.inf
    A[9, 3, 3], A[9, 4, 4] = np.inf, -np.inf
    A[10] = 0.0
    A[11] *= 2.0 ** -1050
    dA = torch.from_numpy(A).cuda()
    P, st, L = _lib.ptr, torch.cuda.current_stream().cuda_stream, _lib.load()
    out = []
    for flags in (0, _lib.WANT_LU):
        det, sign, logabs = (torch.full((12,), 7.0, dtype=torch.float64, device="cuda") for _ in range(3))
        info = torch.full((12,), -1, dtype=torch.int32, device="cuda")
        LU, piv = torch.empty_like(dA), torch.zeros(12, n, dtype=torch.int32, device="cuda")
        rc = L.nppb_d_linalg_batched(12, n, 0, flags | _lib.WANT_DET | _lib.WANT_SLOGDET, P(dA), None, None, None, P(det),
                                     P(sign), P(logabs), P(LU) if flags else None, P(piv) if flags else None, P(info), st)
        assert rc == _lib.OK
        out.append([t.cpu().numpy() for t in (info, det, sign, logabs)])
    for a, b in zip(out[0], out[1]):
        if a.dtype == np.int32:
            np.testing.assert_array_equal(a, b)
        else:
            np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
            np.testing.assert_array_equal(np.isinf(a), np.isinf(b))
