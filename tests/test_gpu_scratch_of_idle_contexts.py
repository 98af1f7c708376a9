"""A state of one context that does not fit takes the scratch of products that another, idle
context keeps: with the device filled up to 128 MiB, 208 MiB come from the residue planes of
the other one's earlier product, which works again afterwards."""
import ctypes as C

import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


def test_state_takes_the_scratch_of_another_context():
    n = 2048
    busy, other = imps.Context(0), imps.Context(0)
    a = torch.randn(n, n, dtype=torch.complex128, device="cuda")
    c, held = torch.empty_like(a), C.c_int64()
    torch.cuda.synchronize()

    def product():   # column-major views: c^T = a^T a^T
        L.check(busy.lib.imps_zgemm(busy.h, 0, 0, n, n, n, 1.0, 0.0, a.data_ptr(), n, a.data_ptr(), n, 0.0, 0.0,
                                    c.data_ptr(), n), busy.h)
        want = a @ a
        return float(torch.linalg.vector_norm(c - want) / torch.linalg.vector_norm(want))

    def workspace():
        L.check(busy.lib.imps_ctx_workspace_bytes(busy.h, C.byref(held)), busy.h)
        return held.value

    assert product() < 1e-13
    before = workspace()
    assert before > 300 << 20
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - (128 << 20), dtype=torch.uint8, device="cuda")
    psi = imps.CanonicalIMPS(other, [4], [1024])   # 3 x 64 MiB and 16 MiB
    assert workspace() < before - (300 << 20)
    del filler, psi
    torch.cuda.empty_cache()
    assert product() < 1e-13
    busy.close()
    other.close()
