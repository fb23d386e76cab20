"""Backward error of the FP64 solves on matrices whose diagonal blocks of U (and of
L, for kept factors) are ill-conditioned: covariance kernels with jitter, random
triangles, Vandermonde matrices.

Bar: Gaussian elimination with partial pivoting and substitution solves
(A + E) x = b with |E| <= 3 n eps |L||U| (Higham, Accuracy and Stability,
theorem 9.4); |L||U| stays within a small multiple of |A| for all of these, so the
normwise backward error is held to 8 n eps, however ill-conditioned A is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def torch(lib):
    import torch
    return torch


def matrices(n):
    rng = np.random.default_rng(n)
    t = np.linspace(0.0, 1.0, n)
    kernel = np.exp(-50.0 * (t[:, None] - t) ** 2)
    out = [kernel + j * np.eye(n) for j in (1e-6, 1e-8, 1e-10)]
    out.append(rng.standard_normal((n, n)))
    if n <= 300:  # the solutions of larger ones leave FP64's range
        out.append(np.triu(rng.standard_normal((n, n))))
    if n <= 64:
        out.append(np.vander(t))
    return np.stack(out)


def rhs(A, k):
    B = np.random.default_rng(k).standard_normal((len(A), A.shape[1], k))
    B[:, :, 0] = A.sum(axis=2)
    return B


def backward_error(A, X, B):
    """Largest over the right-hand sides, per system; residuals in extended precision."""
    out = []
    for a, x, b in zip(A, X, B):
        r = np.abs(a.astype(np.longdouble) @ x.astype(np.longdouble) - b).max(axis=0)
        out.append(float((r / (np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0))).max()))
    return np.array(out)


def check(A, X, B, what):
    err = backward_error(A, X, B)
    assert (err <= 8 * A.shape[1] * EPS).all(), (what, A.shape[1], err)


@pytest.mark.parametrize("n", [33, 40, 64, 200, 257, 512, 513, 1025])
@pytest.mark.parametrize("k", [1, 12, 33])
def test_solve_and_inverse(torch, n, k):
    from numpp_b200 import device
    A = matrices(n)
    B = rhs(A, k)
    dA = torch.from_numpy(A).cuda()
    X, info = device.solve(dA, torch.from_numpy(B).cuda(), check=False)
    assert not info.any()
    check(A, X.cpu().numpy(), B, "solve")
    if k == 1:
        check(A, device.inv(dA).cpu().numpy(), np.broadcast_to(np.eye(n), A.shape), "inv")


@pytest.mark.parametrize("n", [40, 64, 513])
@pytest.mark.parametrize("k", [1, 9, 33])
def test_pivots_at_the_ends_of_the_range(torch, n, k):
    """Diagonal systems whose pivots' reciprocals overflow or are subnormal: the quotients are
    in range, and each is one or two roundings away from its value."""
    from numpp_b200 import device
    d = np.ones((2, n))
    d[0, 3], d[1, 0], d[:, n - 1] = 2.0 ** 1020, 2.0 ** 1023, 2.0 ** -1070
    x = np.random.default_rng(n).integers(1, 8, (2, n, k)).astype(float) / 8
    A = np.zeros((2, n, n))
    A[:, range(n), range(n)] = d
    X, info = device.solve(torch.from_numpy(A).cuda(), torch.from_numpy(d[:, :, None] * x).cuda(), check=False)
    assert not info.any()
    np.testing.assert_allclose(X.cpu().numpy(), x, rtol=2 * EPS)


@pytest.mark.parametrize("n", [40, 64, 200, 513])
@pytest.mark.parametrize("k", [1, 20])
def test_kept_factors(torch, n, k):
    from numpp_b200 import _lib
    A = matrices(n)
    if n <= 64:  # its own factor L, and an ill-conditioned one
        A = np.concatenate([A, [np.eye(n) - np.tril(np.ones((n, n)), -1)]])
    B = rhs(A, k)
    c = len(A)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    LU, X = torch.empty_like(dA), torch.empty_like(dB)
    piv, info = (torch.zeros(s, dtype=torch.int32, device="cuda") for s in ((c, n), (c,)))
    P, st, L = _lib.ptr, torch.cuda.current_stream().cuda_stream, _lib.load()
    assert L.nppb_d_linalg_batched(c, n, 0, _lib.WANT_LU, P(dA), None, None, None, None, None, None, P(LU), P(piv),
                                   P(info), st) == _lib.OK
    assert L.nppb_d_getrs_batched(c, n, k, P(LU), P(piv), P(dB), P(X), st) == _lib.OK
    assert not info.any()
    check(A, X.cpu().numpy(), B, "getrs")


def test_plan(lib):
    from numpp_b200 import _lib
    from numpp_b200.grouped import solve_grouped
    mats = [a for n in (33, 40, 64, 200, 512) for a in matrices(n)]
    n = np.array([len(a) for a in mats], np.int32)
    nrhs = np.array([(1, 8, 32)[i % 3] for i in range(len(mats))], np.int32)
    B = [rhs(a[None], k)[0] for a, k in zip(mats, nrhs)]
    nn, nb = n.astype(np.int64) ** 2, n.astype(np.int64) * nrhs
    off = [np.concatenate([[0], np.cumsum(x)[:-1]]) for x in (nn, nb)]
    sys = {"n": n, "nrhs": nrhs, "a_off": off[0], "b_off": off[1], "inv_off": off[0], "inv_size": int(nn.sum()),
           "A": np.concatenate([a.ravel() for a in mats]), "B": np.concatenate([b.ravel() for b in B])}
    X, inv, _, _, _, info = solve_grouped(sys, _lib.WANT_SOLVE | _lib.WANT_INV)
    assert not info.any()
    for i, a in enumerate(mats):
        x = X[off[1][i]:off[1][i] + nb[i]].reshape(n[i], nrhs[i])
        check(a[None], x[None], B[i][None], "plan %d" % i)
        y = inv[off[0][i]:off[0][i] + nn[i]].reshape(n[i], n[i])
        check(a[None], y[None], np.eye(n[i])[None], "plan's inverse %d" % i)


@pytest.mark.parametrize("n", [64, 200, 512])
def test_mixed_fallback(lib, n):
    """The FP64 solve behind a refinement that stalls meets the tolerance that it always met."""
    from numpp_b200.mixed import solve_mixed
    A = matrices(n)[:4]
    B = rhs(A, 2)
    X, rep = solve_mixed(A, B, tol=8 * n * EPS, max_iter=5)
    assert rep["fallback"][2] and not rep["info"].any()
    check(A, X, B, "mixed")


@pytest.mark.parametrize("n,k,count", [(1030, 2048, 4), (1030, 1984, 4), (2080, 2400, 1), (2080, 2401, 1)])
def test_many_right_hand_sides(torch, n, k, count):
    """Both sides of the rule that hands calls with very many columns to the step kernels (orders
    above 1024). The residual is taken in FP64, which adds (n + 2) eps: 10 n eps in all."""
    from numpp_b200 import _lib, device
    A = torch.from_numpy(matrices(n)[:count]).cuda()
    B = torch.from_numpy(rhs(A.cpu().numpy(), k)).cuda()

    def bound(X, B):
        r = (A @ X - B).abs().amax(dim=1)
        scale = A.abs().sum(dim=2).amax(dim=1)[:, None] * X.abs().amax(dim=1) + B.abs().amax(dim=1)
        assert bool((r <= 10 * n * EPS * scale).all()), float((r / scale).max())

    X, info = device.solve(A, B, check=False)
    assert not info.any()
    bound(X, B)
    X = device.inv(A)
    bound(X, torch.eye(n, dtype=torch.float64, device="cuda").expand_as(A))
    P, st, L = _lib.ptr, torch.cuda.current_stream().cuda_stream, _lib.load()
    LU, Y = torch.empty_like(A), B.clone()
    piv, info = (torch.zeros(s, dtype=torch.int32, device="cuda") for s in ((count, n), (count,)))
    assert L.nppb_d_linalg_batched(count, n, 0, _lib.WANT_LU, P(A), None, None, None, None, None, None, P(LU), P(piv),
                                   P(info), st) == _lib.OK
    assert L.nppb_d_getrs_batched(count, n, k, P(LU), P(piv), P(Y), P(Y), st) == _lib.OK  # in place
    bound(Y, B)


def test_many_right_hand_sides_of_kept_factors(torch):
    from numpp_b200 import _lib
    P, st, L = _lib.ptr, torch.cuda.current_stream().cuda_stream, _lib.load()
    for n, k in ((3008, 2880), (3008, 2912)):
        A = torch.from_numpy(matrices(n)[:1]).cuda()
        B = torch.randn(1, n, k, dtype=torch.float64, device="cuda")
        LU, X = torch.empty_like(A), torch.empty_like(B)
        piv, info = (torch.zeros(s, dtype=torch.int32, device="cuda") for s in ((1, n), (1,)))
        assert L.nppb_d_linalg_batched(1, n, 0, _lib.WANT_LU, P(A), None, None, None, None, None, None, P(LU), P(piv),
                                       P(info), st) == _lib.OK
        assert L.nppb_d_getrs_batched(1, n, k, P(LU), P(piv), P(B), P(X), st) == _lib.OK
        r = (A @ X - B).abs().amax(dim=1)
        scale = A.abs().sum(dim=2).amax(dim=1)[:, None] * X.abs().amax(dim=1) + B.abs().amax(dim=1)
        assert bool((r <= 10 * n * EPS * scale).all())


def test_many_right_hand_sides_under_capture(torch):
    """Captured twice, the calls replay to what they give outside (the re-solve takes its general
    form there, so its digits may differ)."""
    from numpp_b200 import _lib, device
    P, L = _lib.ptr, _lib.load()
    n, k, count = 1030, 2048, 16
    A = torch.from_numpy(matrices(n)[:4]).cuda().repeat(4, 1, 1)
    A.diagonal(dim1=1, dim2=2).add_(1.0)
    B = torch.randn(count, n, k, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    LU = torch.empty_like(A)
    piv, info = (torch.zeros(s, dtype=torch.int32, device="cuda") for s in ((count, n), (count,)))
    assert L.nppb_d_linalg_batched(count, n, 0, _lib.WANT_LU, P(A), None, None, None, None, None, None, P(LU), P(piv),
                                   P(info), st) == _lib.OK
    X = torch.zeros(2, count, n, k, dtype=torch.float64, device="cuda")

    def calls():
        s = torch.cuda.current_stream().cuda_stream
        assert L.nppb_d_getrs_batched(count, n, k, P(LU), P(piv), P(B), P(X[0]), s) == _lib.OK, _lib.last_error()
        assert L.nppb_d_linalg_batched(count, n, k, _lib.WANT_SOLVE, P(A), P(B), P(X[1]), None, None, None, None, None,
                                       None, P(info), s) == _lib.OK, _lib.last_error()

    calls()
    torch.cuda.synchronize()
    want = X.clone()
    for _ in range(2):
        X.zero_()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            calls()
        graph.replay()
        torch.cuda.synchronize()
        for x, w in zip(X, want):
            r = (A @ x - B).abs().amax()
            scale = A.abs().sum(dim=2).amax() * x.abs().amax() + B.abs().amax()
            assert bool(r <= 10 * n * EPS * scale)
        assert torch.equal(X[1], want[1])
