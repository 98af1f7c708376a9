"""The slicing kernels of the split engine at the edges of their tiles (32 lines x 64 k, 4
lines a block, lines too long for a block, ragged ends) for every layout and slice count:
integers below 64 have one or two leading digits, so the products of all slices kept are
exact, and the lines' scales may differ by powers of two.  The AC application collects the
row maxima of its intermediate in the level mix; it agrees with FP64 to the engine's bound."""
import ctypes as C

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, complex).T)).cuda()


@pytest.mark.parametrize("opA,opB", [(0, 0), (2, 0), (0, 2), (2, 2)])
@pytest.mark.parametrize("s", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("M,N,K", [(64, 8192, 65), (129, 300, 1000), (257, 66, 4000), (200, 1000, 193)])
def test_integer_products(opA, opB, s, M, N, K):
    rng = np.random.default_rng(M + N + K)
    X = (rng.integers(-60, 61, (M, K)) + 1j * rng.integers(-60, 61, (M, K))) * 2.0 ** rng.integers(-30, 30, (M, 1))
    Y = (rng.integers(-60, 61, (K, N)) + 1j * rng.integers(-60, 61, (K, N))) * 2.0 ** rng.integers(-30, 30, (1, N))
    A = X if opA == 0 else X.conj().T
    B = Y if opB == 0 else Y.conj().T
    ctx = imps.Context(0, precision=L.IMPS_PREC_SPLIT_I8, nslices=s)
    n0 = ctx.counters()["split_launches"]
    dA, dB = _dev(A), _dev(B)
    dC = torch.full((N, M), np.nan, dtype=torch.complex128, device="cuda")
    L.check(ctx.lib.imps_zgemm(ctx.h, opA, opB, M, N, K, 1.0, 0.0, C.c_void_p(dA.data_ptr()), A.shape[0],
                               C.c_void_p(dB.data_ptr()), B.shape[0], 0.0, 0.0, C.c_void_p(dC.data_ptr()), M), ctx.h)
    assert ctx.counters()["split_launches"] > n0
    assert np.array_equal(dC.cpu().numpy().T, X @ Y)
    ctx.close()


@pytest.mark.parametrize("model,D", [("tfim", 260), ("xxz", 193), ("hubbard", 130)])
def test_ac_with_collected_maxima(model, D):
    W = {"tfim": imps.tfim_hamiltonian(), "xxz": imps.heisenberg_hamiltonian(), "hubbard": imps.hubbard_hamiltonian()}
    H = W[model]
    rng = np.random.default_rng(D)
    m, d = H.Ws[0].shape[0], H.Ws[0].shape[1]

    def rc(*s):
        return np.asfortranarray(rng.standard_normal(s) + 1j * rng.standard_normal(s))
    GL, GR, x = rc(D, m, D), rc(D, m, D), rc(D, d, D)
    y = []
    for s in (0, 5):
        ctx = imps.Context(0) if s == 0 else imps.Context(0, precision=L.IMPS_PREC_SPLIT_I8, nslices=s)
        psi = imps.CanonicalIMPS(ctx, [d], [D])
        envs = imps.DMRGCache(psi, H, build=False)
        envs.set_leftenv(1, GL)
        envs.set_rightenv(1, GR)
        h = imps.AC_hamiltonian(1, psi, H, psi, envs)
        y.append(h(x))
        y.append(h(np.asfortranarray(1e6 * x)) / 1e6)  # other maxima in the same buffers
        ctx.close()
    # two products, each within 16 2^-7s of its lines' scales (at most 6 times their rms here)
    tol = 2 * 16 * 2.0 ** -35 * 36
    for z in y[2:]:
        assert np.linalg.norm(z - y[0]) <= tol * np.linalg.norm(y[0])
