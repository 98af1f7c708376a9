"""A bounded wait that runs out is reported by the call whose product gave up, not by a later
one; only the two asynchronous applications leave it to the next call, whichever that is.  The
waits are made to run out by a one-cycle bound at a size whose products go to the residue
engine."""
import ctypes as C

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu
D = 512


@pytest.fixture()
def setup():
    ctx = imps.Context(0)
    H1 = imps.heisenberg_hamiltonian()
    H = imps.SparseIMPO(H1.Ws * 2)
    rng = np.random.default_rng(3)
    sites = [np.asfortranarray(rng.standard_normal((D, 2, D)) + 1j * rng.standard_normal((D, 2, D))) for _ in range(2)]
    psi = imps.CanonicalIMPS.from_sites(sites, ctx=ctx)
    envs = imps.DMRGCache(psi, H)
    yield ctx, H, psi, envs
    del envs, psi
    ctx.close()


def _limit(ctx, cycles):
    L.check(ctx.lib.imps_ctx_set_wait_limit(ctx.h, cycles), ctx.h)


def test_an_asynchronous_application_reports_at_the_next_call(setup):
    ctx, H, psi, envs = setup
    x = torch.from_numpy(np.ascontiguousarray(psi.AC[0].transpose(2, 1, 0))).cuda()
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    h = H.handle(ctx)
    _limit(ctx, 1)
    assert ctx.lib.imps_ac_apply_dev(envs.h, h, 0, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())) == L.IMPS_OK
    assert ctx.lib.imps_state_copy(psi.h, psi.h) == L.IMPS_TIMEOUT
    _limit(ctx, 0)
    assert ctx.lib.imps_ctx_synchronize(ctx.h) == L.IMPS_OK


@pytest.mark.parametrize("call", ["envs_build", "tdvp_step", "gauge_step"])
def test_the_call_itself_reports(setup, call):
    ctx, H, psi, envs = setup
    _limit(ctx, 1)
    with pytest.raises(L.ImpsError) as e:
        if call == "envs_build":
            envs.build(psi, H)
        elif call == "tdvp_step":
            imps.timestep(psi, H, -0.01j, envs=envs)
        else:
            L.check(ctx.lib.imps_gauge_step(psi.h, 1e-12, 20, None), ctx.h)
    assert e.value.status == L.IMPS_TIMEOUT
    _limit(ctx, 0)
    assert ctx.lib.imps_ctx_synchronize(ctx.h) == L.IMPS_OK   # nothing left behind


def test_a_result_that_gave_up_is_nan(setup):
    """For a caller that waits on its own stream and does not ask for the status."""
    ctx, H, psi, envs = setup
    x = torch.from_numpy(np.ascontiguousarray(psi.AC[0].transpose(2, 1, 0))).cuda()
    y, z = torch.empty_like(x), torch.empty_like(x)
    torch.cuda.synchronize()

    def apply(out):
        return ctx.lib.imps_ac_apply_dev(envs.h, H.handle(ctx), 0, C.c_void_p(x.data_ptr()), C.c_void_p(out.data_ptr()))
    _limit(ctx, 1)
    assert apply(y) == L.IMPS_OK
    torch.cuda.synchronize()
    assert torch.isnan(y.real).all() and torch.isnan(y.imag).all()
    _limit(ctx, 0)
    assert ctx.lib.imps_ctx_synchronize(ctx.h) == L.IMPS_TIMEOUT
    assert apply(z) == L.IMPS_OK and ctx.lib.imps_ctx_synchronize(ctx.h) == L.IMPS_OK
    assert torch.isfinite(torch.view_as_real(z)).all()
