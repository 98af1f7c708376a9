"""Large FP64 products whose outputs exceed one panel of columns: a plane of a panel's
residues stays within 32 MiB, so 8192 rows take 4096 columns at a time.  Integers, exact in every element
(against the same product of another library), with the last panel full, one column wide and
ragged; and in the last panel's columns lines that are summed in FP64: a graded one, which keeps
the FP64 bound, and one with a NaN."""
import ctypes as C

import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu
M, K, PANEL = 8192, 320, 4096


def _ints(g, *s):
    x = torch.randint(-2**18, 2**18, (*s, 2), generator=g, device="cuda").to(torch.float64)
    return torch.view_as_complex(x)


@pytest.mark.parametrize("N,opB", [(2 * PANEL, 0), (PANEL + 1, 0), (PANEL + 333, 1), (2 * PANEL + 70, 0)])
@pytest.mark.parametrize("beta", [0.0, 1.0])
def test_column_panels(N, opB, beta):
    g = torch.Generator(device="cuda").manual_seed(N)
    At, Bt = _ints(g, K, M), _ints(g, N, K)      # rows are the columns of column-major A and B
    C0 = _ints(g, N, M)
    want = Bt @ At + beta * C0                   # (A B)^T
    grade = torch.exp2(-torch.linspace(0, 60, K, device="cuda", dtype=torch.float64))
    At[:, 17] *= grade
    Bt[N - 1] *= grade.flip(0)
    Bt[PANEL, 3] = float("nan")
    stored = Bt if opB == 0 else Bt.T.contiguous()
    out = C0.clone() if beta else torch.full_like(C0, float("nan"))
    ctx = imps.Context(0)
    torch.cuda.synchronize()
    k0 = ctx.counters()["kernels"]
    L.check(ctx.lib.imps_zgemm(ctx.h, 0, opB, M, N, K, 1.0, 0.0, C.c_void_p(At.data_ptr()), M,
                               C.c_void_p(stored.data_ptr()), K if opB == 0 else N, beta, 0.0,
                               C.c_void_p(out.data_ptr()), M), ctx.h)
    assert ctx.counters()["kernels"] - k0 == 2 + 2 * -(-N // PANEL)
    assert torch.isnan(out[PANEL].real).all()
    rows = torch.ones(N, dtype=torch.bool, device="cuda")
    rows[PANEL] = rows[N - 1] = False
    cols = torch.ones(M, dtype=torch.bool, device="cuda")
    cols[17] = False
    assert torch.equal(out[rows][:, cols], want[rows][:, cols])
    # the main lines: n = K terms of an FP64 sum, (K + 1) 2^-53 sum |a| |b| a component, on
    # either side
    for got, a, b, c in ((out[N - 1], At, Bt[N - 1:], C0[N - 1:]), (out[rows][:, 17], At[:, 17:18], Bt[rows], C0[rows][:, 17:18])):
        if N - 1 == PANEL and b.shape[0] == 1:
            continue   # the one column of the last panel holds the NaN
        ref = (b @ a + beta * c).flatten()
        bound = 3 * (K + 2) * 2.0**-53 * (b.abs() @ a.abs() + beta * c.abs()).flatten()
        assert torch.all((got - ref).abs() <= bound)
    ctx.close()
