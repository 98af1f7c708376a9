"""Lines with an infinity or a NaN in a large FP64 product: their elements are plain FP64 sums,
taken a warp each while they are few in a 64 x 16 tile of C and by the whole block otherwise
(the limit is 64), in time of the order of an FP64 product's.  They are what the FP64 tensor
cores make of them (the same call under a workspace cap; alpha multiplies as a complex number,
so an infinite sum ends as a NaN); every other element keeps the bound of the operands'
rounding."""
import ctypes as C

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _gemm(ctx, tA, tB, tC, M, N, K, opA, opB, kernels=4):
    k0 = ctx.counters()["kernels"]
    L.check(ctx.lib.imps_zgemm(ctx.h, opA, opB, M, N, K, 1.0, 0.0, C.c_void_p(tA.data_ptr()), M if opA == 0 else K,
                               C.c_void_p(tB.data_ptr()), K if opB == 0 else N, 0.0, 0.0, C.c_void_p(tC.data_ptr()), M),
            ctx.h)
    assert ctx.counters()["kernels"] - k0 == kernels


@pytest.mark.parametrize("opA,opB", [(0, 0), (1, 1), (0, 1), (1, 0)])
@pytest.mark.parametrize("rows", [[3], [64, 65, 66, 67], [64, 65, 66, 67, 68], list(range(100, 200))])
def test_infinite_lines(opA, opB, rows):
    M, N, K = 513, 520, 700
    rng = np.random.default_rng(len(rows))
    X = rng.integers(-2**20, 2**20, (M, K)) + 1j * rng.integers(-2**20, 2**20, (M, K))
    Y = rng.integers(1, 2**20, (K, N)) * rng.choice([-1, 1], (K, N)) + 1j * rng.integers(1, 2**20, (K, N))
    ks = rng.integers(0, K, len(rows))
    X[rows, ks] = np.inf
    tA, tB = ((torch.from_numpy(np.ascontiguousarray(Z.T if op == 0 else Z)).cuda()) for Z, op in ((X, opA), (Y, opB)))
    tC = torch.empty((N, M), dtype=torch.complex128, device="cuda")
    ctx = imps.Context(0)
    _gemm(ctx, tA, tB, tC, M, N, K, opA, opB)
    got = tC.cpu().numpy().T
    L.check(ctx.lib.imps_ctx_set_workspace_limit(ctx.h, 1), ctx.h)
    _gemm(ctx, tA, tB, tC, M, N, K, opA, opB, kernels=1)
    assert np.array_equal(got[rows], tC.cpu().numpy().T[rows], equal_nan=True) and not np.isfinite(got[rows]).any()
    clean = np.setdiff1d(np.arange(M), rows)
    bound = (np.sqrt(2.0 * K) * 2.0**-57 + 2.0**-51) * np.linalg.norm(X[clean], axis=1)[:, None] * np.linalg.norm(Y, axis=0)
    assert np.all(np.abs(got[clean] - X[clean] @ Y) <= bound)
    ctx.close()


def test_an_all_nan_operand_takes_the_time_of_an_fp64_product():
    n = 2048
    a = torch.full((n, n), float("nan"), dtype=torch.complex128, device="cuda")
    b = torch.randn(n, n, dtype=torch.complex128, device="cuda")
    c = torch.empty_like(a)
    ctx = imps.Context(0)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    _gemm(ctx, a, b, c, n, n, n, 0, 0)
    t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    t0.record()
    _gemm(ctx, a, b, c, n, n, n, 0, 0)
    t1.record()
    torch.cuda.synchronize()
    assert torch.isnan(c.real).all() and torch.isnan(c.imag).all()
    assert t0.elapsed_time(t1) < 8.0 * n**3 / 4e12 * 1e3   # 4 TFLOP/s, a tenth of the FP64 pipe
    ctx.close()
