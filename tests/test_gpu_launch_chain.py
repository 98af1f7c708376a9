"""Kernels placed while the one before them still runs: a chain of asynchronous applications,
each reading what the last one wrote, gives the bits of applications that are waited for, on
the context's stream, on the caller's and from a captured graph.  Normalising between them is
left to the inputs: the operators are scaled so that 40 applications neither grow nor vanish."""
import ctypes as C

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _problem(D, slices):
    ctx = imps.Context(0) if not slices else imps.Context(0, precision=L.IMPS_PREC_SPLIT_I8, nslices=slices)
    H = imps.heisenberg_hamiltonian()
    m, d = H.Ws[0].shape[0], H.Ws[0].shape[1]
    rng = np.random.default_rng(D)

    def rc(*s):
        return np.asfortranarray(rng.standard_normal(s) + 1j * rng.standard_normal(s)) / np.sqrt(2 * m * D)
    psi = imps.CanonicalIMPS(ctx, [d], [D])
    envs = imps.DMRGCache(psi, H, build=False)
    envs.set_leftenv(1, rc(D, m, D))
    envs.set_rightenv(1, rc(D, m, D))
    x = torch.from_numpy(np.ascontiguousarray(rc(D, d, D).T)).cuda()
    torch.cuda.synchronize()

    def apply(a, b):
        L.check(ctx.lib.imps_ac_apply_dev(envs.h, H.handle(ctx), 0, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr())),
                ctx.h)
    return ctx, apply, x, (psi, envs, H)


@pytest.mark.parametrize("D,slices", [(12, 0), (65, 0), (128, 0), (260, 0), (260, 4)])
@pytest.mark.parametrize("where", ["own", "caller", "default"])
def test_chain_has_the_bits_of_single_calls(D, slices, where):
    ctx, apply, x, keep = _problem(D, slices)
    s = torch.cuda.Stream() if where == "caller" else torch.cuda.default_stream()
    if where != "own":
        L.check(ctx.lib.imps_ctx_set_stream(ctx.h, C.c_void_p(s.cuda_stream)), ctx.h)
    n = 40
    one, chain = [x.clone()], [x.clone()] + [torch.empty_like(x) for _ in range(n)]
    torch.cuda.synchronize()
    for _ in range(n):
        y = torch.empty_like(x)
        apply(one[-1], y)
        ctx.synchronize()
        one.append(y)
    for a, b in zip(chain, chain[1:]):
        apply(a, b)
    ctx.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(one, chain))
    assert torch.isfinite(torch.view_as_real(chain[-1])).all() and chain[-1].abs().max() > 0
    ctx.close()


@pytest.mark.parametrize("D", [12, 65, 128])
def test_captured_chain(D):
    ctx, apply, x, keep = _problem(D, 0)
    s = torch.cuda.Stream()
    L.check(ctx.lib.imps_ctx_set_stream(ctx.h, C.c_void_p(s.cuda_stream)), ctx.h)
    ys, zs = ([x.clone()] + [torch.empty_like(x) for _ in range(6)] for _ in range(2))
    torch.cuda.synchronize()
    for a, b in zip(ys, ys[1:]):
        apply(a, b)
    ctx.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        for a, b in zip(zs, zs[1:]):
            apply(a, b)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    # no scratch may be allocated while capturing, so a product can be summed in another order
    tol = 6 * 4 * 2 * D * 2.0 ** -53
    assert all(torch.linalg.norm(a - b) <= tol * torch.linalg.norm(a) for a, b in zip(ys, zs))
    del g
    ctx.close()
