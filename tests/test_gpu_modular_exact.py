"""Large FP64 products whose result is a double are exact, as an FP64 sum is: integer operands
with lines of 2-norm up to 2^57 convert without rounding, their product's residues determine it,
and the reconstruction rounds once.  Small sums between large terms, zeros, sums near 2^53, and
powers of two on the lines; sums beyond 2^53 are rounded to the nearest double."""
import ctypes as C

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = imps.Context(0)
    yield c
    c.close()


def _gemm(ctx, X, Y, opA=0):
    M, K = X.shape
    N = Y.shape[1]
    A = X if opA == 0 else X.conj().T
    tA, tB = (torch.from_numpy(np.ascontiguousarray(Z.T)).cuda() for Z in (A, Y))
    tC = torch.empty((N, M), dtype=torch.complex128, device="cuda")
    k0 = ctx.counters()["kernels"]
    L.check(ctx.lib.imps_zgemm(ctx.h, opA, 0, M, N, K, 1.0, 0.0, C.c_void_p(tA.data_ptr()), A.shape[0],
                               C.c_void_p(tB.data_ptr()), K, 0.0, 0.0, C.c_void_p(tC.data_ptr()), M), ctx.h)
    assert ctx.counters()["kernels"] - k0 == 4
    return tC.cpu().numpy().T


def _ints(rng, b, *s):
    return rng.integers(-2**b, 2**b + 1, s) + 1j * rng.integers(-2**b, 2**b + 1, s)


@pytest.mark.parametrize("bits", [1, 8, 20, 21])
@pytest.mark.parametrize("M,N,K,opA", [(512, 512, 768, 0), (700, 511, 1921, 2), (1025, 300, 640, 0)])
def test_integer_products(ctx, bits, M, N, K, opA):
    rng = np.random.default_rng(bits + K)
    X, Y = _ints(rng, bits, M, K), _ints(rng, bits, K, N)
    assert np.array_equal(_gemm(ctx, X, Y, opA), X @ Y)


def test_cancelling_sums_and_scales(ctx):
    rng = np.random.default_rng(4)
    M, N, K = 600, 520, 800
    X, Y = _ints(rng, 20, M, K), _ints(rng, 20, K, N)
    X[:, K // 2:] = X[:, : K // 2]
    Y[K // 2:] = -Y[: K // 2]          # every sum cancels
    Y[7, ::3] += 1                     # but for one product
    rs, cs = 2.0 ** rng.integers(-200, 200, M)[:, None], 2.0 ** rng.integers(-200, 200, N)
    want = (X @ Y) * rs * cs
    assert np.array_equal(_gemm(ctx, X * rs, Y * cs), want)
    assert np.count_nonzero(want) == np.count_nonzero((X[:, 7, None] != 0) & (np.arange(N) % 3 == 0)[None])


def test_long_sums_are_rounded_to_the_nearest_double(ctx):
    """Real and imaginary parts of up to 80 bits, summed in Python integers."""
    rng = np.random.default_rng(9)
    M, N, K, rows = 512, 512, 640, 12
    X, Y = _ints(rng, 35, M, K), _ints(rng, 34, K, N)
    got = _gemm(ctx, X, Y)[:rows]
    for part in range(2):
        for i in range(rows):
            for j in range(0, N, 37):
                a = [(int(z.real), int(z.imag)) for z in X[i]]
                b = [(int(z.real), int(z.imag)) for z in Y[:, j]]
                if part == 0:
                    v = sum(p[0] * q[0] - p[1] * q[1] for p, q in zip(a, b))
                else:
                    v = sum(p[0] * q[1] + p[1] * q[0] for p, q in zip(a, b))
                g = got[i, j].real if part == 0 else got[i, j].imag
                assert abs(int(g) - v) <= 2.0**-53 * abs(v) * (1 + 2.0**-40)
