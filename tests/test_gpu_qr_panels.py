"""QRpos at the row counts where the panel kernel changes its shape (128, 256, 512, 1024,
2048, 4096 rows) and where a panel or an outer block is ragged: Q R = M, Q isometric and R
upper triangular with a positive diagonal, each to the backward error of Householder QR
(a small multiple of sqrt(n) eps); a matrix with dependent and zero columns keeps Q R = M;
split-mode and FP64 contexts agree to the same bound although they sum differently."""
import numpy as np
import pytest

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def ctxs():
    c = [imps.Context(0), imps.Context(0, precision=L.IMPS_PREC_SPLIT_I8, nslices=-1)]
    yield c
    for x in c:
        x.close()


@pytest.mark.parametrize("m,n", [(1, 1), (15, 17), (128, 16), (129, 33), (256, 65), (257, 64), (512, 130), (513, 48),
                                 (1024, 70), (1025, 64), (2049, 40), (4096, 17), (4097, 20)])
def test_panels(ctxs, m, n):
    rng = np.random.default_rng(m + n)
    M = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    k = min(m, n)
    tol = 40 * np.sqrt(k) * EPS
    R0 = None
    for ctx in ctxs:
        Q, R = imps.qrpos(M, ctx=ctx)
        assert np.linalg.norm(Q @ R - M) <= tol * np.linalg.norm(M)
        assert np.linalg.norm(Q.conj().T @ Q - np.eye(k)) <= tol * np.sqrt(k)
        assert np.array_equal(np.tril(R[:, :k], -1), np.zeros((k, k)))
        d = np.diag(R)
        assert np.all(d.real > 0) and np.all(np.abs(d.imag) <= 4 * EPS * d.real)
        if R0 is not None:
            cond = np.linalg.cond(M[:, :k])
            assert np.linalg.norm(R - R0) <= 2 * tol * cond * np.linalg.norm(M)
        R0 = R


@pytest.mark.parametrize("m,n", [(256, 64), (600, 96)])
def test_dependent_and_zero_columns(ctxs, m, n):
    rng = np.random.default_rng(2)
    M = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    M[:, 5] = 0.0
    M[:, 20] = M[:, 3]
    M[:, 40] = 1j * M[:, 7] - M[:, 21]
    for ctx in ctxs:
        Q, R = imps.qrpos(M, ctx=ctx)
        assert np.linalg.norm(Q @ R - M) <= 40 * np.sqrt(n) * EPS * np.linalg.norm(M)
