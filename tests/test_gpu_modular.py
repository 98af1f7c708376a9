"""The FP64 GEMM in residue arithmetic on the int8 tensor cores.  An element may be off by
the rounding of the scaled operands (sqrt(K / 2) against lines of 2-norm at least 2^57, on
each side) and the final conversion: (sqrt(2 K) 2^-57 + 2^-51) ||a_i|| ||b_j||.  The inputs
are integers below 2^20, whose products numpy sums exactly."""
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


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, complex).T)).cuda()


def _op(X, op):
    return X if op == 0 else X.T if op == 1 else X.conj().T


def _gemm(ctx, A, B, opA, opB, C0=None, alpha=1.0 + 0j, beta=0j, kernels=4):
    M, K = _op(A, opA).shape
    N = _op(B, opB).shape[1]
    dA, dB = _dev(A), _dev(B)
    dC = torch.full((N, M), np.nan, dtype=torch.complex128, device="cuda") if C0 is None else _dev(C0)
    k0 = ctx.counters()["kernels"]
    L.check(ctx.lib.imps_zgemm(ctx.h, opA, opB, M, N, K, alpha.real, alpha.imag, C.c_void_p(dA.data_ptr()), A.shape[0],
                               C.c_void_p(dB.data_ptr()), B.shape[0], beta.real, beta.imag,
                               C.c_void_p(dC.data_ptr()), M), ctx.h)
    if kernels:
        assert ctx.counters()["kernels"] - k0 == kernels  # norms, planes, products, reconstruction
    return dC.cpu().numpy().T


def _ints(rng, *shape):
    return rng.integers(-2**20, 2**20, shape) + 1j * rng.integers(-2**20, 2**20, shape)


def _bound(X, Y):
    K = X.shape[1]
    return (np.sqrt(2.0 * K) * 2.0**-57 + 2.0**-51) * np.linalg.norm(X, axis=1)[:, None] * np.linalg.norm(Y, axis=0)


@pytest.mark.parametrize("opA,opB", [(0, 0), (0, 1), (0, 2), (1, 0), (1, 1), (2, 0), (2, 2)])
@pytest.mark.parametrize("M,N,K", [(512, 512, 768), (513, 257, 1025), (255, 1100, 1000), (1025, 300, 640),
                                   (700, 511, 1921)])
def test_products_within_the_rounding_of_the_operands(ctx, opA, opB, M, N, K):
    rng = np.random.default_rng(M + 7 * N + K)
    X, Y = _ints(rng, M, K), _ints(rng, K, N)
    got = _gemm(ctx, _op(X, opA), _op(Y, opB), opA, opB)
    assert np.all(np.abs(got - X @ Y) <= _bound(X, Y))


def test_alpha_beta_and_scales_far_from_one(ctx):
    rng = np.random.default_rng(5)
    M, N, K = 600, 520, 800
    X, Y = _ints(rng, M, K), _ints(rng, K, N)
    C0 = _ints(rng, M, N)
    got = _gemm(ctx, X, Y, 0, 0, C0, 2 - 1j, 0.5 + 3j)
    ref = (2 - 1j) * (X @ Y) + (0.5 + 3j) * C0
    assert np.all(np.abs(got - ref) <= 3 * _bound(X, Y) + 2.0**-50 * np.abs(ref))
    # lines whose squares leave the double range, and lines of zeros
    rs = np.where(np.arange(M) % 3 == 0, 2.0**-700, np.where(np.arange(M) % 3 == 1, 2.0**600, 1.0))
    X2 = X * rs[:, None]
    X2[7] = 0.0
    got = _gemm(ctx, X2, Y, 0, 0)
    assert np.all(got[7] == 0.0)
    with np.errstate(all="ignore"):
        assert np.all(np.abs(got / rs[:, None] - (X2 / rs[:, None]) @ Y) <= 8 * _bound(X, Y))


@pytest.mark.parametrize("where", ["a", "b"])
def test_nan_and_inf_reach_the_elements_they_reach_in_fp64(ctx, where):
    rng = np.random.default_rng(6)
    M, N, K = 600, 520, 800
    X, Y = _ints(rng, M, K), _ints(rng, K, N)
    if where == "a":
        X[3, 5] = np.inf
        X[300, 799] = np.nan
    else:
        Y[5, 3] = -np.inf
        Y[799, 300] = 1j * np.nan
    got = _gemm(ctx, X, Y, 0, 0)
    hit = ~np.isfinite(X).all(axis=1)[:, None] | ~np.isfinite(Y).all(axis=0)[None, :]
    assert not np.isfinite(got[hit]).any()
    clean = ~hit
    Xf, Yf = np.where(np.isfinite(X), X, 0), np.where(np.isfinite(Y), Y, 0)
    assert np.all(np.abs(got - Xf @ Yf)[clean] <= _bound(Xf, Yf)[clean])
    ctx.synchronize()


def test_without_scratch_the_fp64_tensor_cores_answer(ctx):
    rng = np.random.default_rng(7)
    X, Y = _ints(rng, 512, 768), _ints(rng, 768, 512)
    L.check(ctx.lib.imps_ctx_set_workspace_limit(ctx.h, 1 << 20), ctx.h)
    got = _gemm(ctx, X, Y, 0, 0, kernels=1)
    L.check(ctx.lib.imps_ctx_set_workspace_limit(ctx.h, 0), ctx.h)
    assert np.array_equal(got, X @ Y)


def test_bounded_wait_runs_out_and_context_recovers():
    """A one-cycle bound: a wait of a CTA pair gives up, both CTAs' copies land before either
    leaves, the status comes with the synchronisation, and the context goes on."""
    c = imps.Context(0)
    rng = np.random.default_rng(5)
    A = rng.integers(-9, 10, (1100, 900)) + 1j * rng.integers(-9, 10, (1100, 900))
    B = rng.integers(-9, 10, (900, 700)) + 1j * rng.integers(-9, 10, (900, 700))
    L.check(c.lib.imps_ctx_set_wait_limit(c.h, 1), c.h)
    for _ in range(3):
        with pytest.raises(L.ImpsError) as e:
            _gemm(c, A, B, 0, 0)
            c.synchronize()
        assert e.value.status == L.IMPS_TIMEOUT
    L.check(c.lib.imps_ctx_set_wait_limit(c.h, 0), c.h)
    assert np.linalg.norm(_gemm(c, A, B, 0, 0) - A @ B) <= 1e-14 * np.linalg.norm(A) * np.linalg.norm(B)
    c.close()
