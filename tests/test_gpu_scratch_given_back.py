"""Scratch that only makes products faster is given back when a state does not fit beside it:
with the device filled up to 128 MiB, a state of 208 MiB comes from the residue planes of an
earlier product, and the product still works afterwards."""
import ctypes as C

import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


def test_state_takes_the_scratch_of_products():
    n = 2048
    ctx = imps.Context(0)
    a = torch.randn(n, n, dtype=torch.complex128, device="cuda")
    c, held = torch.empty_like(a), C.c_int64()
    torch.cuda.synchronize()

    def product():   # column-major views: c^T = a^T a^T
        L.check(ctx.lib.imps_zgemm(ctx.h, 0, 0, n, n, n, 1.0, 0.0, a.data_ptr(), n, a.data_ptr(), n, 0.0, 0.0,
                                   c.data_ptr(), n), ctx.h)
        want = a @ a
        return float(torch.linalg.vector_norm(c - want) / torch.linalg.vector_norm(want))

    def workspace():
        L.check(ctx.lib.imps_ctx_workspace_bytes(ctx.h, C.byref(held)), ctx.h)
        return held.value

    assert product() < 1e-13
    before = workspace()
    assert before > 300 << 20
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - (128 << 20), dtype=torch.uint8, device="cuda")
    psi = imps.CanonicalIMPS(ctx, [4], [1024])   # 3 x 64 MiB and 16 MiB
    assert workspace() < before - (300 << 20)
    del filler, psi
    torch.cuda.empty_cache()
    assert product() < 1e-13
