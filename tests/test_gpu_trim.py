"""Device memory that a context keeps between calls is counted and can be had back: blocks of
destroyed states (up to 256 MiB) and the scratch of large products, by a workspace cap, under
which neither is kept, and by a trim, after which both are kept again."""
import ctypes as C

import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu
STATE = 3 * 16 * 4 * 256 * 256 + 16 * 256 * 256   # AL, AR, AC and C at D = 256, d = 4


@pytest.fixture()
def ctx():
    c = imps.Context(0)
    yield c
    c.close()


def _held(ctx):
    b = C.c_int64()
    L.check(ctx.lib.imps_ctx_workspace_bytes(ctx.h, C.byref(b)), ctx.h)
    return b.value


def _state(ctx):
    psi = imps.CanonicalIMPS(ctx, [4], [256])
    del psi


def _product(ctx):
    n = 1024
    a = torch.ones(n, n, dtype=torch.complex128, device="cuda")
    c = torch.empty_like(a)
    torch.cuda.synchronize()
    L.check(ctx.lib.imps_zgemm(ctx.h, 0, 0, n, n, n, 1.0, 0.0, a.data_ptr(), n, a.data_ptr(), n, 0.0, 0.0, c.data_ptr(),
                               n), ctx.h)
    assert torch.all(c == n)


def test_blocks_of_destroyed_states(ctx):
    before = _held(ctx)
    _state(ctx)
    assert _held(ctx) == before + STATE
    _state(ctx)                       # the same blocks
    assert _held(ctx) == before + STATE
    ctx.trim()
    assert _held(ctx) == before
    _state(ctx)
    L.check(ctx.lib.imps_ctx_set_workspace_limit(ctx.h, 1 << 40), ctx.h)
    assert _held(ctx) == before
    _state(ctx)
    assert _held(ctx) == before       # nothing is kept under a cap
    L.check(ctx.lib.imps_ctx_set_workspace_limit(ctx.h, 0), ctx.h)
    _state(ctx)
    assert _held(ctx) == before + STATE


def test_scratch_of_products(ctx):
    _product(ctx)
    full = _held(ctx)
    assert full > 64 << 20
    free = torch.cuda.mem_get_info()[0]
    ctx.trim()
    assert _held(ctx) < full - (64 << 20)
    assert torch.cuda.mem_get_info()[0] >= free + (64 << 20)
    _product(ctx)
    assert _held(ctx) == full
