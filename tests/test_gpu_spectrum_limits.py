"""The entanglement spectrum under workspace caps: the matrix with one column of padding at most,
its column norms and a flag are enough (whole blocks of 16 columns are used where they fit),
and a cap below that is IMPS_OOM.  The values agree with numpy to the backward error of a
one-sided Jacobi sweep."""
import ctypes as C

import numpy as np
import pytest

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _state(ctx, Cm):
    psi = imps.CanonicalIMPS(ctx, [2], [Cm.shape[0]])
    psi.set(L.IMPS_C, 0, np.asfortranarray(Cm))
    return psi


@pytest.mark.parametrize("D", [1, 2, 17, 18, 20, 33])
def test_smallest_cap(D):
    rng = np.random.default_rng(D)
    Cm = rng.standard_normal((D, D)) + 1j * rng.standard_normal((D, D))
    want = np.linalg.svd(Cm, compute_uv=False) ** 2
    want /= want.sum()
    P = D + D % 2
    need = 16 * D * P + 8 * P + 64
    for cap in (need, 0, need - 1):
        ctx = imps.Context(0)
        psi = _state(ctx, Cm)
        L.check(ctx.lib.imps_ctx_set_workspace_limit(ctx.h, cap), ctx.h)
        if cap == need - 1:
            with pytest.raises(Exception) as e:
                imps.entanglement_spectrum(psi, 1)
            assert getattr(e.value, "status", None) == -3 or isinstance(e.value, MemoryError)
        else:
            got = imps.entanglement_spectrum(psi, 1)
            assert np.all(np.abs(got - want) <= 50 * np.sqrt(D) * np.finfo(float).eps * want[0])
        del psi
        ctx.close()


@pytest.mark.parametrize("exponent", [-530, -300, 0, 300, 510, 511])
def test_squares_near_the_ends_of_the_range(exponent):
    """A matrix of rank two whose leading squared singular value is 1.7 4^exponent."""
    D = 20
    Cm = np.zeros((D, D), complex)
    Cm[3, 5] = np.sqrt(1.7) * 2.0**exponent
    Cm[4, 6] = 0.5j * np.sqrt(1.7) * 2.0**exponent
    ctx = imps.Context(0)
    psi = _state(ctx, Cm)
    got = imps.entanglement_spectrum(psi, 1)
    assert np.all(np.abs(got - np.r_[0.8, 0.2, np.zeros(D - 2)]) <= 8 * np.finfo(float).eps)
    del psi
    ctx.close()
