"""Scales of the residue products' operands: a line's integers have 2-norm in [2^57, 2^58]
whatever its magnitude, so the rounding of the operands is a random sum of size
sqrt(1/6 + 1/6) 2^-57 ||a_i|| ||b_j|| (both lines' elements off by at most 1/2 in each
component, independently), also for lines whose squares leave the double range and for lines
that one element dominates.  The reference is summed in 80-bit arithmetic; eight standard
deviations, and the rounding of the result."""
import ctypes as C

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opA", [0, 1])
@pytest.mark.parametrize("exponent", [-1000, -700, -466, 0, 460, 500])
@pytest.mark.parametrize("K", [1024, 8192])
def test_lines_of_every_scale(opA, exponent, K):
    M, N, rows = 512, 256, 6
    rng = np.random.default_rng(K + exponent)

    def rc(*s):
        return rng.standard_normal(s) + 1j * rng.standard_normal(s)
    X, Y = rc(M, K), rc(K, N)
    X[:4] *= 1e-5
    X[0, 3] = 1.0            # one element carries the line: in the first chunk of K,
    X[1, K - 1] = 1.0 - 0.5j     # in the last,
    X[2, K // 2] = -1.0          # in the middle
    X[3] *= np.exp2(np.linspace(0, 60, K))   # growing along K, the chunks' sums on both sides of the range
    S = np.full(M, 2.0 ** exponent)
    dA = X * S[:, None]
    dA, Xs = (dA if opA == 0 else dA.T), dA[:rows]
    tA, tB = (torch.from_numpy(np.ascontiguousarray(Z.T)).cuda() for Z in (dA, Y))
    tC = torch.empty((N, M), dtype=torch.complex128, device="cuda")
    ctx = imps.Context(0)
    k0 = ctx.counters()["kernels"]
    L.check(ctx.lib.imps_zgemm(ctx.h, opA, 0, M, N, K, 1.0, 0.0, C.c_void_p(tA.data_ptr()), dA.shape[0],
                               C.c_void_p(tB.data_ptr()), K, 0.0, 0.0, C.c_void_p(tC.data_ptr()), M), ctx.h)
    assert ctx.counters()["kernels"] - k0 == 4
    got = tC.cpu().numpy().T[:rows] / 2.0 ** exponent
    Xs = Xs / 2.0 ** exponent
    ref = Xs.astype(np.clongdouble) @ Y.astype(np.clongdouble)
    na, nb = np.linalg.norm(Xs, axis=1)[:, None], np.linalg.norm(Y, axis=0)
    bound = 8 * np.sqrt(1 / 3) * 2.0**-57 * na * nb + 2.0**-51 * np.abs(ref)
    assert np.all(np.abs((got - ref).astype(complex)) <= bound)
    ctx.close()
