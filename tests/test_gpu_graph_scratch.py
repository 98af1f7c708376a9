"""A captured chain of effective-Hamiltonian applications is replayed after other calls on the
context have grown, capped and given back the scratch that products use: the graph holds none
of it, so every replay gives the bits of the first.  (The products of these sizes share their
K stages through such scratch when they are not captured.)"""
import ctypes as C

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [65, 128])
def test_replays_after_the_scratch_has_gone(D):
    ctx = imps.Context(0)
    s = torch.cuda.Stream()
    L.check(ctx.lib.imps_ctx_set_stream(ctx.h, C.c_void_p(s.cuda_stream)), ctx.h)
    H = imps.heisenberg_hamiltonian()
    m, d = H.Ws[0].shape[0], H.Ws[0].shape[1]
    rng = np.random.default_rng(D)

    def rc(*shape):
        return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) / np.sqrt(2 * m * D)
    psi = imps.CanonicalIMPS(ctx, [d], [D])
    envs = imps.DMRGCache(psi, H, build=False)
    envs.set_leftenv(1, rc(D, m, D))
    envs.set_rightenv(1, rc(D, m, D))
    x = torch.from_numpy(np.ascontiguousarray(rc(D, d, D).T)).cuda()
    y = torch.empty_like(x)

    def apply(out):
        L.check(ctx.lib.imps_ac_apply_dev(envs.h, H.handle(ctx), 0, C.c_void_p(x.data_ptr()), C.c_void_p(out.data_ptr())),
                ctx.h)

    def product(M, N, K):
        a, b = (torch.ones(k, dtype=torch.complex128, device="cuda") for k in (M * K, K * N))
        c = torch.empty(M * N, dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        L.check(ctx.lib.imps_zgemm(ctx.h, 0, 0, M, N, K, 1.0, 0.0, C.c_void_p(a.data_ptr()), M, C.c_void_p(b.data_ptr()),
                                   K, 0.0, 0.0, C.c_void_p(c.data_ptr()), M), ctx.h)
        assert torch.all(c == K)

    apply(torch.empty_like(x))   # the buffers of an application of this size
    ctx.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        apply(y)
    g.replay()
    torch.cuda.synchronize()
    first = y.clone()
    assert torch.isfinite(torch.view_as_real(first)).all()
    for step in (lambda: product(64, 64, 4000), lambda: product(200, 190, 5000),
                 lambda: L.check(ctx.lib.imps_ctx_set_workspace_limit(ctx.h, 1 << 40), ctx.h)):
        step()
        filler = torch.full((1 << 25,), np.nan, dtype=torch.float64, device="cuda")   # takes what was freed
        y.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, first)
        del filler
    del g
    ctx.close()
