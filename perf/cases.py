"""The work that users of this framework have it do, as timed cases.

Every case goes through a public entry point: ``numpp_b200.device`` for torch
stacks, ``numpp_b200.grouped.Plan`` for uneven batches, and the C ABI
(include/numpp_b200.h) for the calls that have no Python front end on device
buffers (solve and det from one factorisation, the mixed-precision solve,
re-solves on kept factors, least squares). Inputs are device-resident, drawn
from the seed with torch's generator; right-hand sides and matrices are N(0,1)
with n added to the diagonal, as ``numpp_b200.workloads`` draws them, except
where a case says otherwise.

``listed`` holds the cases, ``draw`` draws more from the ranges they stand
for, ``prepare`` makes what a program has in hand before the call, ``run`` is
one call, ``work`` its bytes and operations, ``exact`` its result as torch
gives it in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from numpp_b200 import _lib, device, workloads
from numpp_b200.grouped import Plan

P = _lib.ptr
UNEVEN_FLAGS = _lib.WANT_SOLVE | _lib.WANT_SLOGDET | _lib.WANT_INV


def listed():
    return [
        # Many tiny systems, solution and determinant from one factorisation:
        # the circuit / per-pixel batch. One launch, so launches count.
        {"name": "solve_det_256x32", "op": "solve_det", "count": 256, "n": 32, "nrhs": 1},
        # One system in single precision: the plain solve(a, b) of a script.
        {"name": "solve_1x300_f32", "op": "solve", "count": 1, "n": 300, "nrhs": 1, "dtype": "float32"},
        # An uneven batch in a kept plan: solve and slogdet of every system, the
        # inverse of a tenth of them. The framework's headline workload. `orders`
        # draws the orders and right-hand-side counts, the seed the entries.
        {"name": "uneven_8192", "op": "uneven", "count": 8192, "n_lo": 4, "n_hi": 512, "orders": 2025},
        # A uniform stack of middling systems.
        {"name": "solve_64x1024", "op": "solve", "count": 64, "n": 1024, "nrhs": 1, "dtype": "float64"},
        # The largest order served.
        {"name": "solve_8x4096", "op": "solve", "count": 8, "n": 4096, "nrhs": 1, "dtype": "float64"},
        # Inverses of a stack whose order is no multiple of anything.
        {"name": "inv_400x201", "op": "inv", "count": 400, "n": 201, "dtype": "float64"},
        # FP32 factors with FP64 refinement, to FP64 accuracy: a middling stack,
        # and a few large systems of an odd order with several right-hand sides.
        {"name": "mixed_64x1024", "op": "mixed", "count": 64, "n": 1024, "nrhs": 1, "log_kappa": 4.0},
        {"name": "mixed_5x3001", "op": "mixed", "count": 5, "n": 3001, "nrhs": 8, "log_kappa": 2.0},
        # Covariance factors.
        {"name": "cholesky_512x256", "op": "cholesky", "count": 512, "n": 256, "dtype": "float64"},
        # New right-hand sides on factors kept from an earlier call, as a time
        # stepper or a server does.
        {"name": "getrs_48x777", "op": "getrs", "count": 48, "n": 777, "nrhs": 16},
        # Many regressions of one shape.
        {"name": "lstsq_1024x200x32", "op": "lstsq", "count": 1024, "m": 200, "n": 32, "nrhs": 1},
        # The stacked product that matrix_power and its callers rest on.
        {"name": "matmul_1024x128", "op": "matmul", "count": 1024, "m": 128, "k": 128, "n": 128,
         "dtype": "float64"},
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], even over its logarithm."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _count(rng, most, values, each):
    """A stack size of at most `most` matrices whose entries stay within `values`."""
    return _log(rng, 1, max(1, min(most, int(values / each))))


def draw(rng):
    op = rng.choice(["solve_det", "solve", "solve", "uneven", "uneven", "inv", "mixed", "mixed", "cholesky",
                     "getrs", "lstsq", "matmul"])
    dtype = rng.choice(["float64", "float64", "float64", "float32"])
    if op == "solve_det":
        n = _log(rng, 3, 64)
        return {"op": op, "count": _log(rng, 16, 4096), "n": n, "nrhs": rng.choice([1, 1, 2, 5, 8])}
    if op == "solve":
        n = _log(rng, 8, 4096)
        return {"op": op, "count": _count(rng, 2048, 1.0e8, n * n), "n": n, "nrhs": rng.choice([1, 1, 3, 8, 32, 64]),
                "dtype": dtype}
    if op == "uneven":
        hi = _log(rng, 32, 1024)
        return {"op": op, "count": _log(rng, 64, 8192 if hi <= 512 else 1024), "n_lo": 4, "n_hi": hi,
                "orders": rng.randrange(1 << 30)}
    if op == "inv":
        n = _log(rng, 8, 1024)
        return {"op": op, "count": _count(rng, 2048, 4.0e7, n * n), "n": n, "dtype": dtype}
    if op == "mixed":
        n = _log(rng, 100, 4096)
        return {"op": op, "count": _count(rng, 512, 1.0e8, n * n), "n": n, "nrhs": rng.choice([1, 1, 2, 4, 8]),
                "log_kappa": rng.uniform(1.0, 4.0)}
    if op == "cholesky":
        n = _log(rng, 8, 2048)
        return {"op": op, "count": _count(rng, 2048, 6.0e7, n * n), "n": n, "dtype": dtype}
    if op == "getrs":
        n = _log(rng, 16, 4096)
        return {"op": op, "count": _count(rng, 512, 6.0e7, n * n), "n": n, "nrhs": rng.choice([1, 2, 7, 16, 32, 64])}
    if op == "lstsq":
        n = _log(rng, 2, 64)
        m = _log(rng, n, max(n, min(512, (26000 - n * n) // n)))
        return {"op": op, "count": _log(rng, 16, 1024), "m": m, "n": n, "nrhs": rng.choice([1, 1, 4, 8])}
    m, k, n = (_log(rng, 16, 1024) for _ in range(3))
    return {"op": op, "count": _count(rng, 2048, 4.0e7, max(m * k, k * n, m * n)), "m": m, "k": k, "n": n,
            "dtype": dtype}


def _randn(g, *shape):
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)


def _shifted(g, count, n):
    A = _randn(g, count, n, n)
    A.diagonal(dim1=1, dim2=2).add_(float(n))
    return A


def _orthogonal(g, count, n):
    """Orthogonal factors of N(0,1) matrices, by Cholesky QR."""
    G = _randn(g, count, n, n)
    R = torch.linalg.cholesky(G.transpose(1, 2) @ G, upper=True)
    return torch.linalg.solve_triangular(R, G, upper=True, left=False)


def _conditioned(g, count, n, kappa):
    """Q1 diag(sigma) Q2^T, sigma log-spaced from 1 to kappa: workloads.conditioned_batch on the GPU."""
    sigma = torch.logspace(0.0, math.log10(kappa), n, dtype=torch.float64, device="cuda")
    return ((_orthogonal(g, count, n) * sigma) @ _orthogonal(g, count, n).transpose(1, 2)).contiguous()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _ok(rc):
    if rc != _lib.OK:
        raise RuntimeError("status %d: %s" % (rc, _lib.last_error()))


def _orders(case):
    """The packed layout of workloads.uneven_batch without its entries."""
    rng = np.random.default_rng(case["orders"])
    count, lo, hi = case["count"], case["n_lo"], case["n_hi"]
    n = np.clip(np.floor(np.exp(rng.uniform(np.log(lo), np.log(hi + 1), size=count))), lo, hi).astype(np.int32)
    nrhs = rng.choice(np.asarray([1, 8, 32], np.int32), size=count).astype(np.int32)
    nn, nb = n.astype(np.int64) ** 2, n.astype(np.int64) * nrhs
    want = rng.random(count) < 0.1
    inv = np.where(want, nn, 0)

    def start(sizes):
        return np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int64)

    return {"n": n, "nrhs": nrhs, "a_off": start(nn), "b_off": start(nb), "count": count,
            "inv_off": np.where(want, start(inv), -1).astype(np.int64), "a_size": int(nn.sum()),
            "b_size": int(nb.sum()), "inv_size": int(inv.sum())}


def _uneven(case, g):
    """An uneven batch, its entries drawn on the GPU."""
    sys = _orders(case)
    n = sys["n"].astype(np.int64)
    A = _randn(g, sys["a_size"])
    j = np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n)
    diagonal = np.repeat(sys["a_off"], n) + j * np.repeat(n + 1, n)
    A[torch.from_numpy(diagonal).cuda()] += torch.from_numpy(np.repeat(n, n).astype(np.float64)).cuda()
    return sys, A, _randn(g, sys["b_size"])


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    op, count = case["op"], case["count"]
    s = {"case": case}
    dtype = getattr(torch, case.get("dtype", "float64"))
    new = torch.empty
    f64, i32 = {"dtype": torch.float64, "device": "cuda"}, {"dtype": torch.int32, "device": "cuda"}
    if op == "uneven":
        sys, s["A"], s["B"] = _uneven(case, g)
        s["sys"], s["plan"] = sys, Plan(sys, UNEVEN_FLAGS)
        s["X"], s["inv"] = torch.zeros_like(s["B"]), torch.zeros(max(sys["inv_size"], 1), **f64)
        s["sign"], s["logabs"], s["info"] = new(count, **f64), new(count, **f64), new(count, **i32)
    elif op == "matmul":
        s["A"] = _randn(g, count, case["m"], case["k"]).to(dtype)
        s["B"] = _randn(g, count, case["k"], case["n"]).to(dtype)
    elif op == "lstsq":
        m, n, k = case["m"], case["n"], case["nrhs"]
        s["A"], s["B"] = _randn(g, count, m, n), _randn(g, count, m, k)
        s["X"], s["S"], s["resid"] = new(count, n, k, **f64), new(count, min(m, n), **f64), torch.zeros(count, k, **f64)
        s["rank"], s["has"] = new(count, **i32), new(count, **i32)
    elif op == "cholesky":
        W = _randn(g, count, case["n"], case["n"])
        A = W @ W.transpose(1, 2)
        A.diagonal(dim1=1, dim2=2).add_(float(case["n"]))
        s["A"] = A.to(dtype)
    else:
        n = case["n"]
        s["A"] = _conditioned(g, count, n, 10.0 ** case["log_kappa"]) if op == "mixed" else _shifted(g, count, n).to(dtype)
        if op != "inv":
            s["B"] = _randn(g, count, n, case["nrhs"]).to(dtype)
        if op in ("solve_det", "mixed", "getrs"):
            s["X"], s["info"] = torch.empty_like(s["B"]), torch.zeros(count, **i32)
        if op == "solve_det":
            s["det"] = new(count, **f64)
        if op == "mixed":
            s["berr"], s["iters"], s["fallback"] = new(count, **f64), new(count, **i32), new(count, **i32)
        if op == "getrs":  # the factors a program keeps
            s["LU"], s["piv"] = torch.empty_like(s["A"]), new(count, n, **i32)
            _ok(_lib.load().nppb_d_linalg_batched(count, n, 0, _lib.WANT_LU, P(s["A"]), None, None, None, None, None,
                                                  None, P(s["LU"]), P(s["piv"]), P(s["info"]), _stream()))
    return s


def run(s):
    c = s["case"]
    op = c["op"]
    if op == "solve":
        return device.solve(s["A"], s["B"], check=False)
    if op == "inv":
        return device.inv(s["A"], check=False)
    if op == "cholesky":
        return device.cholesky(s["A"], check=False)
    if op == "matmul":
        return device.matmul_batched(s["A"], s["B"])
    if op == "uneven":
        s["plan"].execute(s["A"], s["B"], s["X"], s["inv"], None, s["sign"], s["logabs"], s["info"], _stream())
        return s["X"], s["inv"], s["sign"], s["logabs"], s["info"]
    L = _lib.load()
    if op == "solve_det":
        _ok(L.nppb_d_linalg_batched(c["count"], c["n"], c["nrhs"], _lib.WANT_SOLVE | _lib.WANT_DET, P(s["A"]),
                                    P(s["B"]), P(s["X"]), None, P(s["det"]), None, None, None, None, P(s["info"]),
                                    _stream()))
        return s["X"], s["det"], s["info"]
    if op == "getrs":
        _ok(L.nppb_d_getrs_batched(c["count"], c["n"], c["nrhs"], P(s["LU"]), P(s["piv"]), P(s["B"]), P(s["X"]),
                                   _stream()))
        return s["X"]
    if op == "lstsq":
        _ok(L.nppb_d_lstsq_batched(c["count"], c["m"], c["n"], c["nrhs"], P(s["A"]), P(s["B"]), -1.0, P(s["X"]),
                                   P(s["S"]), P(s["rank"]), P(s["resid"]), P(s["has"]), _stream()))
        return s["X"], s["S"], s["resid"], s["rank"], s["has"]
    # A tolerance of 1e-14 asks for a solution as good as the FP64 solve's. How many
    # corrections that took, and the backward error left, tell of the way there.
    _ok(L.nppb_d_solve_mixed_batched(c["count"], c["n"], c["nrhs"], P(s["A"]), P(s["B"]), P(s["X"]), None, 1e-14, 30, 0,
                                     P(s["info"]), P(s["berr"]), None, P(s["iters"]), P(s["fallback"]), _stream()))
    return s["X"], s["fallback"]


def work(case):
    """LAPACK's operation counts; each input read once and each output written once."""
    op, count = case["op"], case["count"]
    if op == "uneven":
        sys = _orders(case)
        return {"bytes": workloads.uneven_bytes(sys), "flops": workloads.uneven_flops(sys)}
    size = 4 if case.get("dtype") == "float32" else 8
    n, k = case["n"], case.get("nrhs", 0)
    if op == "matmul":
        m, q = case["m"], case["k"]
        return {"bytes": size * count * (m * q + q * n + m * n), "flops": 2.0 * count * m * q * n}
    if op == "lstsq":  # by a QR factorisation and the SVD of its triangle
        m = case["m"]
        return {"bytes": 8 * count * (m * n + m * k + n * k + n + k),
                "flops": count * (2.0 * m * n * n + 4.0 * m * n * k + 11.0 * n ** 3)}
    lu, sub = float(workloads.lu_flops(n)), float(workloads.getrs_flops(n, k))
    if op == "getrs":
        return {"bytes": count * (8 * n * n + 4 * n + 16 * n * k), "flops": count * sub}
    if op == "cholesky":  # the lower triangle in, the whole factor out
        return {"bytes": size * count * (n * (n + 1) // 2 + n * n), "flops": count * n ** 3 / 3.0}
    if op == "inv":
        return {"bytes": size * count * 2 * n * n, "flops": count * 2.0 * n ** 3}
    return {"bytes": size * count * (n * n + 2 * n * k), "flops": count * (lu + sub)}


def exact(case, seed):
    s = prepare(case, seed)
    op = case["op"]
    if op == "uneven":
        sys, A, B = s["sys"], s["A"], s["B"]
        X, inv = torch.zeros_like(B), torch.zeros_like(s["inv"])
        sign, logabs = torch.zeros_like(s["sign"]), torch.zeros_like(s["logabs"])

        def at(offsets, size):
            return (torch.as_tensor(offsets, device="cuda")[:, None] + torch.arange(size, device="cuda")).reshape(-1)

        for n in np.unique(sys["n"]):
            n, who = int(n), np.nonzero(sys["n"] == n)[0]
            M = A[at(sys["a_off"][who], n * n)].view(-1, n, n)
            i = torch.as_tensor(who, device="cuda")
            sign[i], logabs[i] = torch.linalg.slogdet(M)
            for k in (1, 8, 32):
                of = np.nonzero(sys["nrhs"][who] == k)[0]
                if len(of):
                    b = at(sys["b_off"][who[of]], n * k)
                    X[b] = torch.linalg.solve(M[torch.as_tensor(of, device="cuda")], B[b].view(-1, n, k)).reshape(-1)
            of = np.nonzero(sys["inv_off"][who] >= 0)[0]
            if len(of):
                inv[at(sys["inv_off"][who[of]], n * n)] = torch.linalg.inv(M[torch.as_tensor(of, device="cuda")]).reshape(-1)
        return X, inv, sign, logabs, None
    A = s["A"].double()
    B = s["B"].double() if "B" in s else None
    if op == "matmul":
        return A @ B
    if op == "inv":
        return torch.linalg.inv(A), None
    if op == "cholesky":
        return torch.linalg.cholesky(A), None
    if op == "lstsq":
        U, S, Vh = torch.linalg.svd(A, full_matrices=False)
        X = Vh.transpose(1, 2) @ ((U.transpose(1, 2) @ B) / S[:, :, None])
        over = case["m"] > case["n"]
        return X, S, ((A @ X - B) ** 2).sum(dim=1) if over else None, None, None
    X = torch.linalg.solve(A, B)
    if op == "solve_det":
        return X, torch.linalg.det(A), None
    return X if op == "getrs" else (X, None)
