"""The FP64 GEMM with its K stages shared by several CTAs: integer-valued inputs are exact
in FP64 whatever the order of the sum, so the products must be bit-exact; with a workspace
cap the same call runs unshared and gives the same bits."""
import ctypes as C

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, complex).T)).cuda()


def _op(X, op):
    return X if op == 0 else X.T if op == 1 else X.conj().T


@pytest.mark.parametrize("opA,opB", [(0, 0), (2, 0), (0, 2), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 33), (64, 64, 2048), (65, 63, 1031), (3, 200, 4100), (260, 130, 17)])
def test_shared_k_products_bit_exact(opA, opB, M, N, K):
    rng = np.random.default_rng(M + 3 * N + K)
    A = _op(rng.integers(-40, 41, (M, K)) + 1j * rng.integers(-40, 41, (M, K)), opA)
    B = _op(rng.integers(-40, 41, (K, N)) + 1j * rng.integers(-40, 41, (K, N)), opB)
    C0 = (rng.integers(-5, 6, (M + 2, N)) + 1j * rng.integers(-5, 6, (M + 2, N))).astype(complex)
    ref = C0.copy()
    ref[:M] = (2 - 1j) * (_op(A, opA) @ _op(B, opB)) + (1 + 3j) * C0[:M]
    ctx = imps.Context(0)
    for cap in (0, 1):
        L.check(ctx.lib.imps_ctx_set_workspace_limit(ctx.h, cap), ctx.h)
        dA, dB, dC = _dev(A), _dev(B), _dev(C0)
        L.check(ctx.lib.imps_zgemm(ctx.h, opA, opB, M, N, K, 2.0, -1.0, C.c_void_p(dA.data_ptr()), A.shape[0],
                                   C.c_void_p(dB.data_ptr()), B.shape[0], 1.0, 3.0, C.c_void_p(dC.data_ptr()), M + 2),
                ctx.h)
        assert np.array_equal(dC.cpu().numpy().T, ref)
    ctx.close()
