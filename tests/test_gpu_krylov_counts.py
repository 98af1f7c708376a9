"""The matvec that a Krylov solver queues ahead of its host's small problem is not one of the
solve's applications when it is thrown away: the context counts as many as the solver reports,
for solves of one step, of a few and of a whole basis, and results do not depend on it."""
import ctypes as C

import numpy as np
import pytest

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problem():
    D = 48
    ctx = imps.Context(0)
    H1 = imps.heisenberg_hamiltonian(1.0, 0.5)
    H = imps.SparseIMPO(H1.Ws)
    m, d = H1.Ws[0].shape[0], H1.Ws[0].shape[1]
    rng = np.random.default_rng(1)

    def rc(*s):
        return np.asfortranarray(rng.standard_normal(s) + 1j * rng.standard_normal(s))
    psi = imps.CanonicalIMPS(ctx, [d], [D])
    envs = imps.DMRGCache(psi, H, build=False)
    GL, GR = rc(D, m, D) / D, rc(D, m, D) / D
    GL, GR = (np.asfortranarray(X + X.transpose(2, 1, 0).conj()) for X in (GL, GR))
    GL[:, 0, :], GR[:, m - 1, :] = np.eye(D), np.eye(D)
    envs.set_leftenv(1, GL)
    envs.set_rightenv(1, GR)
    yield ctx, H, envs, rc(D, d, D), rc(D, D)
    del envs, psi
    ctx.close()


@pytest.mark.parametrize("tol", [10.0, 0.5, 0.1, 1e-2, 1e-4])
@pytest.mark.parametrize("eager", [0, 1])
def test_eigsolve(problem, tol, eager):
    ctx, H, envs, x0, c0 = problem
    for which, v in (("ac_apply", x0), ("c_apply", c0)):
        out, info = np.zeros_like(v), L.KrylovInfo()
        n0 = ctx.counters()[which]
        if which == "ac_apply":
            ctx.lib.imps_eigsolve_ac(envs.h, H.handle(ctx), 0, L.dptr(v), L.dptr(out), tol, 20, 3, eager, C.byref(info))
        else:
            ctx.lib.imps_eigsolve_c(envs.h, 0, L.dptr(v), L.dptr(out), tol, 20, 3, eager, C.byref(info))
        assert ctx.counters()[which] - n0 == info.numops


@pytest.mark.parametrize("dt", [1e-5, 1e-3, 3e-2])
def test_exponentiate(problem, dt):
    ctx, H, envs, x0, _ = problem
    out, info = np.zeros_like(x0), L.KrylovInfo()
    n0, f0 = ctx.counters()["ac_apply"], ctx.counters()["gemm_flops"]
    ctx.lib.imps_exponentiate_ac(envs.h, H.handle(ctx), 0, 0.0, -dt, L.dptr(x0), L.dptr(out), 1e-10, 20, 5, C.byref(info))
    n, f1 = info.numops, ctx.counters()["gemm_flops"]
    assert ctx.counters()["ac_apply"] - n0 == n
    y = np.zeros_like(x0)
    ctx.lib.imps_ac_apply(envs.h, H.handle(ctx), 0, L.dptr(x0), L.dptr(y))
    assert f1 - f0 == n * (ctx.counters()["gemm_flops"] - f1)


def test_a_solve_of_one_step_runs_no_second_matvec(problem):
    """A basis of one vector cannot have one queued ahead: the same launches."""
    ctx, H, envs, x0, _ = problem
    out, info, used = np.zeros_like(x0), L.KrylovInfo(), []
    for krylovdim in (1, 20):
        for _ in range(2):   # the second without first-use work
            k0 = ctx.counters()["kernels"]
            ctx.lib.imps_eigsolve_ac(envs.h, H.handle(ctx), 0, L.dptr(x0), L.dptr(out), 1e6, krylovdim, 3, 1, C.byref(info))
            assert info.numops == 1
        used.append(ctx.counters()["kernels"] - k0)
    assert used[0] == used[1]
