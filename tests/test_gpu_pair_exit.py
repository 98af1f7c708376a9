"""Residue products on CTA pairs whose second CTA has nothing to write (64 and 128 rows: the
pair's upper 128 rows are padding) and so reaches the end of the kernel first; it stays until
the arrivals of the leader's commits at its barriers are in.  Integer operands: the bound of
the operands' rounding, and the same bits every time."""
import ctypes as C
import re
from pathlib import Path

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L


def test_both_ctas_of_a_pair_wait_for_the_commits_they_receive():
    src = (Path(imps.__file__).parent / "csrc" / "gemm_modular.cu").read_text()
    body = src[src.index("void leave_pair("):]
    body = body[:body.index("\n}\n")]
    # outside the branch of the leader, ahead of the return of the ordinary end
    head = body[:body.index("return;")]
    assert re.search(r"mbar_drain\(b\.drain", head) and not re.search(r"rank == 0", head)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(64, 4096, 2048), (128, 4000, 1500), (129, 3000, 1500)])
def test_thin_products_repeat(M, N, K):
    rng = np.random.default_rng(M)
    X = rng.integers(-2**20, 2**20, (M, K)) + 1j * rng.integers(-2**20, 2**20, (M, K))
    Y = rng.integers(-2**20, 2**20, (K, N)) + 1j * rng.integers(-2**20, 2**20, (K, N))
    dA, dB = (torch.from_numpy(np.ascontiguousarray(Z.T)).cuda() for Z in (X, Y))
    dC = torch.empty((N, M), dtype=torch.complex128, device="cuda")
    ctx = imps.Context(0)
    first = None
    for _ in range(10):
        k0 = ctx.counters()["kernels"]
        L.check(ctx.lib.imps_zgemm(ctx.h, 0, 0, M, N, K, 1.0, 0.0, C.c_void_p(dA.data_ptr()), M, C.c_void_p(dB.data_ptr()),
                                   K, 0.0, 0.0, C.c_void_p(dC.data_ptr()), M), ctx.h)
        if M == 128:   # (the other two are near the line to the FP64 tensor cores)
            assert ctx.counters()["kernels"] - k0 == 4
        got = dC.cpu().numpy().T
        if first is None:
            first = got
            bound = (np.sqrt(2.0 * K) * 2.0**-57 + 2.0**-51) * np.linalg.norm(X, axis=1)[:, None] * np.linalg.norm(Y, axis=0)
            assert np.all(np.abs(got - X @ Y) <= bound)
        assert np.array_equal(got, first)
    ctx.close()
