"""Kernels that write into another CTA's shared memory, launched while another
stream keeps the SMs busy, so that the CTAs of a cluster start at different
times: every result equals the one of a quiet GPU bit for bit (the order of the
operations does not depend on when a CTA starts)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch(lib):
    import torch
    return torch


def calls(torch, n, k):
    """solve (k_sys_solve on 2 to 8 CTAs), kept factors (k_panel above order 512) with
    getrs, and the mixed solve (k_mx_trsv_c), as functions that return new tensors."""
    from numpp_b200 import _lib, device
    L, P = _lib.load(), _lib.ptr
    rng = np.random.default_rng(n)
    A = torch.from_numpy(rng.standard_normal((1, n, n)) + 2 * np.sqrt(n) * np.eye(n)).cuda()
    B = torch.from_numpy(rng.standard_normal((1, n, k))).cuda()

    def stream():
        return torch.cuda.current_stream().cuda_stream

    def kept():
        LU, X = torch.empty_like(A), torch.empty_like(B)
        piv, info = (torch.zeros(s, dtype=torch.int32, device="cuda") for s in ((1, n), (1,)))
        assert L.nppb_d_linalg_batched(1, n, 0, _lib.WANT_LU, P(A), None, None, None, None, None, None, P(LU), P(piv),
                                       P(info), stream()) == _lib.OK
        assert L.nppb_d_getrs_batched(1, n, k, P(LU), P(piv), P(B), P(X), stream()) == _lib.OK
        return X

    def mixed():
        X = torch.empty_like(B)
        info = torch.zeros(1, dtype=torch.int32, device="cuda")
        assert L.nppb_d_solve_mixed_batched(1, n, k, P(A), P(B), P(X), None, 1e-13, 10, 0, P(info), None, None, None,
                                            None, stream()) == _lib.OK
        return X

    return [lambda: device.solve(A, B, check=False)[0], kept, mixed]


@pytest.mark.parametrize("n", [256, 512, 700, 2049])
def test_cluster_ctas_that_start_apart(torch, n):
    fns = calls(torch, n, 5)
    quiet = [f() for f in fns]
    torch.cuda.synchronize()
    M = torch.randn(2048, 2048, device="cuda", dtype=torch.float32)
    busy, work = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(4):
        with torch.cuda.stream(busy):
            for _ in range(20):
                M = M @ M * 1e-3
        with torch.cuda.stream(work):
            got = [f() for f in fns]
        torch.cuda.synchronize()
        for g, q in zip(got, quiet):
            assert torch.equal(g, q)
