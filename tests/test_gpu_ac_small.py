"""The one-launch AC application of small states against a plain einsum and against the
general path (a split-mode context keeps it, and runs products this small in FP64): square
and rectangular bonds from 1 up, column shares that are empty or uneven, every model, an MPO
level without blocks.  Sums of K terms in another order differ by at most about K eps."""
import numpy as np
import pytest

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu
W = {"tfim": imps.tfim_hamiltonian(1.0, 0.7).Ws[0], "xxz": imps.heisenberg_hamiltonian(1.0, 0.3).Ws[0],
     "hubbard": imps.hubbard_hamiltonian().Ws[0]}


def _hole():
    w = np.array(W["xxz"], order="F")
    w[:, :, 2, :] = 0.0
    return w


def _apply(ctx, w, GL, GR, x):
    H = imps.SparseIMPO([w])
    Dl, d, Dr = x.shape
    psi = imps.CanonicalIMPS(ctx, [d, d], [Dr, Dl])
    H = imps.SparseIMPO([w, w])
    envs = imps.DMRGCache(psi, H, build=False)
    envs.set_leftenv(1, GL)
    envs.set_rightenv(1, GR)
    k0 = ctx.counters()["kernels"]
    y = imps.AC_hamiltonian(1, psi, H, psi, envs)(x)
    return y, ctx.counters()["kernels"] - k0


@pytest.mark.parametrize("model", ["tfim", "xxz", "hubbard", "hole"])
@pytest.mark.parametrize("Dl,Dr", [(1, 1), (2, 3), (7, 9), (8, 8), (16, 16), (5, 24), (24, 5), (22, 23), (40, 40)])
def test_small_ac(model, Dl, Dr):
    w = _hole() if model == "hole" else W[model]
    rng = np.random.default_rng(Dl * 50 + Dr)
    d, m = w.shape[1], w.shape[0]

    def rc(*s):
        return np.asfortranarray(rng.standard_normal(s) + 1j * rng.standard_normal(s))
    GL, GR, x = rc(Dl, m, Dl), rc(Dr, m, Dr), rc(Dl, d, Dr)
    t = np.einsum("iujs,bia,asc->bujc", w, GL, x)
    ref = np.einsum("bujc,cjd->bud", t, GR)
    size = np.einsum("bujc,cjd->bud", np.einsum("iujs,bia,asc->bujc", np.abs(w), np.abs(GL), np.abs(x)), np.abs(GR))
    ctx, general = imps.Context(0), imps.Context(0, precision=L.IMPS_PREC_SPLIT_I8, nslices=5)
    y, k = _apply(ctx, w, GL, GR, x)
    z, kg = _apply(general, w, GL, GR, x)
    tol = 4 * (Dl + Dr * m + m * d) * np.finfo(float).eps
    assert np.all(np.abs(y - ref) <= tol * size)
    assert np.all(np.abs(y - z) <= tol * size)
    macs = Dl * Dl * m * d * Dr + Dl * d * Dr * Dr * m
    assert (k == 1) == (macs <= 7e5 and model != "hole")
    assert kg >= 3
    ctx.close()
    general.close()
