"""Batches of small systems on a device that is nearly full. Above order 32 the calls
need no more than the step kernels do, a matrix and 8616 bytes a system (8616 alone
in a caller's workspace): where the system-resident kernels' 512 n bytes more do not
fit, a uniform batch is worked through in parts and a plan takes the step kernels."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SETUP = """
import numpy as np, torch
from numpp_b200 import _lib, device
from numpp_b200.grouped import Plan
L, P = _lib.load(), _lib.ptr
st = torch.cuda.current_stream().cuda_stream
g = torch.Generator(device="cuda")
g.manual_seed(1)
def systems(count, n, k):
    A = torch.randn(count, n, n, dtype=torch.float64, device="cuda", generator=g)
    A.diagonal(dim1=1, dim2=2).add_(float(n))
    return A, torch.randn(count, n, k, dtype=torch.float64, device="cuda", generator=g)
def fill(left):
    # kernels are loaded and the library's pool is empty; leaves `left` bytes
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - left, dtype=torch.uint8, device="cuda")
def check(A, X, B, some):
    r = (A[some] @ X[some] - B[some]).abs().max()
    assert float(r) <= 1e-12 * A.shape[1] * 4, float(r)
"""

CASES = {
    "solve": """
count, n = 60000, 33
A, B = systems(count, n, 1)
X, info = torch.zeros_like(B), torch.full((count,), -1, dtype=torch.int32, device="cuda")
full = fill(1500 << 20)
assert L.nppb_d_linalg_batched(count, n, 1, _lib.WANT_SOLVE, P(A), P(B), P(X), None, None, None, None, None, None,
                               P(info), st) == _lib.OK, _lib.last_error()
torch.cuda.synchronize()
del full
assert not info.any()
check(A, X, B, slice(0, 64)); check(A, X, B, slice(count // 2 - 32, count // 2 + 32)); check(A, X, B, slice(-64, None))
""",
    "workspace": """
count, n = 40000, 64
A, B = systems(count, n, 1)
A0 = A[-64:].clone()
X, info = torch.zeros_like(B), torch.full((count,), -1, dtype=torch.int32, device="cuda")
piv = torch.empty(count, n, dtype=torch.int32, device="cuda")
full = fill(600 << 20)
assert L.nppb_d_linalg_batched(count, n, 1, _lib.WANT_SOLVE, P(A), P(B), P(X), None, None, None, None, P(A), P(piv),
                               P(info), st) == _lib.OK, _lib.last_error()
torch.cuda.synchronize()
del full
assert not info.any()
check(A0, X[-64:], B[-64:], slice(None))
""",
    "getrs": """
count, n = 60000, 33
A, B = systems(count, n, 1)
LU, X = torch.empty_like(A), torch.zeros_like(B)
piv, info = torch.empty(count, n, dtype=torch.int32, device="cuda"), torch.zeros(count, dtype=torch.int32, device="cuda")
half = count // 2  # (the factorisation's own plan is small enough to stay)
for s in (0, half):
    assert L.nppb_d_linalg_batched(half, n, 0, _lib.WANT_LU, P(A[s:]), None, None, None, None, None, None, P(LU[s:]),
                                   P(piv[s:]), P(info[s:]), st) == _lib.OK
full = fill(1000 << 20)
assert L.nppb_d_getrs_batched(count, n, 1, P(LU), P(piv), P(B), P(X), st) == _lib.OK, _lib.last_error()
torch.cuda.synchronize()
del full
check(A, X, B, slice(0, 64)); check(A, X, B, slice(-64, None))
""",
    "plan": """
count, n = 60000, 33
A, B = systems(count, n, 1)
X, info = torch.zeros_like(B), torch.full((count,), -1, dtype=torch.int32, device="cuda")
at = np.arange(count, dtype=np.int64)
sys = {"n": np.full(count, n), "nrhs": np.full(count, 1), "a_off": at * n * n, "b_off": at * n,
       "inv_off": np.full(count, -1)}
full = fill(1500 << 20)
plan = Plan(sys, _lib.WANT_SOLVE)
plan.execute(A, B, X, None, None, None, None, info, st)
torch.cuda.synchronize()
del full
assert not info.any()
check(A, X, B, slice(0, 64)); check(A, X, B, slice(-64, None))
""",
}


@pytest.mark.parametrize("case", CASES)
def test_nearly_full_device(lib, case):
    out = subprocess.run([sys.executable, "-c", SETUP + CASES[case] + "\nprint('fits')"], cwd=ROOT, text=True,
                         capture_output=True, timeout=300)
    assert out.returncode == 0 and "fits" in out.stdout, out.stdout + out.stderr
