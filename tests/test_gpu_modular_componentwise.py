"""Large FP64 products keep the componentwise accuracy of an FP64 sum, whatever the structure of
their operands: with u = 2^-53, n_ij the number of nonzero terms and S_ij = sum_k |a_ik| |b_kj|,
an FP64 sum rounds n times, each by at most u S, and the residue products answer only where
their error (0.41 sqrt(n) u S in the root mean square at the worst) is no larger.  Eight
standard deviations of n independent roundings and those of the result: 8 (sqrt(n) + 1) u S.
Elements without a term are zero, and products with an identity, a permutation or one-term
lines are exact to the product's own rounding.  The reference is summed in 80-bit arithmetic
over some rows and columns (its error, n 2^-64 S, is 2000 times smaller)."""
import ctypes as C

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu
M, N, K = 640, 600, 1024


@pytest.fixture(scope="module")
def ctx():
    c = imps.Context(0)
    yield c
    c.close()


def _rc(rng, *s):
    return rng.standard_normal(s) + 1j * rng.standard_normal(s)


def _case(name):
    rng = np.random.default_rng(11)
    X, Y = _rc(rng, M, K), _rc(rng, K, N)
    grade = np.exp2(-np.linspace(0, 60, K))
    if name == "one_large":            # (2^60, 1, 1, ...) times (0, 1, 1, ...)
        X[:] = 1.0
        X[:, 0] = 2.0**60
        Y[:] = 1.0
        Y[0] = 0.0
    elif name == "identity":           # times columns over 14 decades
        X[:] = np.eye(M, K)
        Y *= 10.0 ** rng.uniform(-14, 0, (K, N))
    elif name == "permutation":
        X[:] = np.eye(K)[rng.permutation(K)][:M]
    elif name == "near_identity":
        X *= 1e-17
        X += np.eye(M, K)
    elif name == "graded":             # the large elements of one side meet the small ones of the other
        X *= grade
        Y *= grade[::-1, None]
    elif name == "graded_rows":        # one side only, some rows
        X[::7] *= grade
    elif name == "graded_alike":
        X *= grade
        Y *= grade[:, None]
    elif name == "wide":
        X *= np.exp(6 * rng.standard_normal((M, K)))
        Y *= np.exp(6 * rng.standard_normal((K, N)))
    elif name == "triangular":
        X = np.triu(_rc(rng, K, K))[K - M:]
        Y = np.tril(Y)
    elif name == "blocks":             # disjoint supports give zeros
        X[: M // 2, K // 2:] = 0
        X[M // 2:, : K // 2] = 0
        Y[K // 2:, : N // 2] = 0
        Y[: K // 2, N // 2:] = 0
    elif name == "sparse":
        X *= rng.random((M, K)) < 0.002
        Y *= rng.random((K, N)) < 0.3
    elif name == "few":                # a handful of elements of a tile only
        X[5] *= grade
        Y[:, 9] *= grade[::-1]
    elif name == "real":
        X, Y = X.real + 0j, Y.real + 0j
    return X, Y


NAMES = ["random", "real", "one_large", "identity", "permutation", "near_identity", "graded", "graded_rows",
         "graded_alike", "wide", "triangular", "blocks", "sparse", "few"]


@pytest.mark.parametrize("opA,opB,beta", [(0, 0, 0.0), (2, 0, 0.0), (0, 2, 1.0), (1, 1, 0.0)])
@pytest.mark.parametrize("name", NAMES)
def test_componentwise(ctx, name, opA, opB, beta):
    X, Y = _case(name)
    rng = np.random.default_rng(3)
    scale = 2.0 ** rng.integers(-300, 300, M)[:, None]   # rows far apart
    X = X * scale
    C0 = _rc(rng, M, N) * scale * 1e-3 if beta else np.full((M, N), np.nan + 0j)

    def stored(Z, op):   # op(stored) = Z
        return Z if op == 0 else Z.T if op == 1 else Z.conj().T
    A, B = stored(X, opA), stored(Y, opB)
    tA, tB, tC = (torch.from_numpy(np.ascontiguousarray(Z.T)).cuda() for Z in (A, B, C0))
    k0 = ctx.counters()["kernels"]
    L.check(ctx.lib.imps_zgemm(ctx.h, opA, opB, M, N, K, 1.0, 0.0, C.c_void_p(tA.data_ptr()), A.shape[0],
                               C.c_void_p(tB.data_ptr()), B.shape[0], beta, 0.0, C.c_void_p(tC.data_ptr()), M), ctx.h)
    assert ctx.counters()["kernels"] - k0 == 4
    got = tC.cpu().numpy().T
    rows = np.unique(np.r_[0:10, rng.integers(0, M, 30), M - 5:M])
    cols = np.unique(np.r_[0:12, rng.integers(0, N, 30), N - 5:N])
    Xs, Ys = X[rows], Y[:, cols]
    ref = (Xs.astype(np.clongdouble)[:, :, None] * Ys.astype(np.clongdouble)[None]).sum(axis=1)
    S = np.abs(Xs) @ np.abs(Ys)
    n = (Xs != 0).astype(float) @ (Ys != 0).astype(float)
    u = 2.0**-53
    got, C0 = got[np.ix_(rows, cols)], C0[np.ix_(rows, cols)]
    bound = 8 * (np.sqrt(n) + 1) * u * S
    if beta:
        ref, bound = ref + C0, bound + 2 * u * (S + np.abs(C0))
    err = np.abs((got - ref).astype(complex))
    assert np.all(err <= bound), (name, float((err / np.maximum(bound, 1e-300)).max()))
    if name in ("identity", "permutation") and not beta:
        assert np.array_equal(got, ref.astype(complex))
    if name == "one_large" and not beta:
        assert np.array_equal(got, ref.astype(complex))
