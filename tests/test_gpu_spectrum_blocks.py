"""Entanglement spectra at the sizes where the block Jacobi changes its shape (blocks of 8
columns, 128 / 256 / 512 rows) against LAPACK: backward-stable singular values are off by a
small multiple of sqrt(D) eps of the largest, so the normalised squares by twice that.  A
workspace cap takes the matrix without the QR and agrees to the same bound."""
import numpy as np
import pytest

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _matrix(kind, D, rng):
    A = rng.standard_normal((D, D)) + 1j * rng.standard_normal((D, D))
    B = rng.standard_normal((D, D)) + 1j * rng.standard_normal((D, D))
    if kind == "decay":
        return (A * np.exp(-16 * np.arange(D) / D)) @ B
    if kind == "graded":
        return A * np.exp(-40 * np.arange(D) / D)
    r = max(1, D // 3)
    return A[:, :r] @ B[:r] * 1e120


@pytest.mark.parametrize("kind", ["decay", "graded", "rank"])
@pytest.mark.parametrize("D", [1, 2, 7, 16, 17, 128, 129, 256, 257, 512, 513])
def test_spectrum(kind, D):
    A = _matrix(kind, D, np.random.default_rng(D))
    q = np.linalg.svd(A / np.abs(A).max(), compute_uv=False) ** 2
    q /= q.sum()
    ctx = imps.Context(0)
    psi = imps.CanonicalIMPS(ctx, [2], [D])
    psi.set(L.IMPS_C, 0, A)
    tol = 40 * np.sqrt(D) * np.finfo(float).eps
    for cap in (0, 1 << 30) if D <= 129 else (0,):
        L.check(ctx.lib.imps_ctx_set_workspace_limit(ctx.h, cap), ctx.h)
        p = imps.entanglement_spectrum(psi, 1)
        assert np.all(np.diff(p) <= 0) and abs(p.sum() - 1) <= tol
        assert np.max(np.abs(p - q)) <= tol
    ctx.close()
