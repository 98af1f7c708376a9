"""IMPS_FP64_ENGINE=2 keeps a context on the FP64 tensor cores: a product that residues would
form in four launches takes one, or two where CTAs share its K stages, which under a workspace
cap become one with the bits of the ordinary context's capped product."""
import ctypes as C

import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _product(ctx, a, b):
    n = a.shape[0]
    c = torch.empty_like(a)
    torch.cuda.synchronize()
    k0 = ctx.counters()["kernels"]
    L.check(ctx.lib.imps_zgemm(ctx.h, 0, 0, n, n, n, 1.0, 0.0, C.c_void_p(a.data_ptr()), n, C.c_void_p(b.data_ptr()), n,
                               0.0, 0.0, C.c_void_p(c.data_ptr()), n), ctx.h)
    return c, ctx.counters()["kernels"] - k0


def test_fp64_tensor_cores_only(monkeypatch):
    a, b = (torch.randn(1024, 1024, dtype=torch.complex128, device="cuda") for _ in range(2))
    out = {}
    for engine in ("0", "2"):
        monkeypatch.setenv("IMPS_FP64_ENGINE", engine)
        ctx = imps.Context(0)
        out[engine] = _product(ctx, a, b)
        L.check(ctx.lib.imps_ctx_set_workspace_limit(ctx.h, 1), ctx.h)
        out[engine, "capped"] = _product(ctx, a, b)
        ctx.close()
    assert out["0"][1] == 4 and out["2"][1] <= 2
    assert out["0", "capped"][1] == out["2", "capped"][1] == 1
    assert torch.equal(out["0", "capped"][0], out["2", "capped"][0])
    bound = 3 * 1026 * 2.0**-53 * (b.abs() @ a.abs())   # column-major views: c = b a
    for c, _ in out.values():
        assert torch.all((c - b @ a).abs() <= bound)
