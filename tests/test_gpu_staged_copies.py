"""Large host arrays (4 MiB and more) are moved by several threads, but their transfers belong
to the context's stream as the calling thread sees it.  With cudaStreamPerThread, whose handle
names another stream in every thread, a transfer comes after the kernels queued before it: an
upload does not overtake applications that still read the buffer, a download not the
application that writes it.  Sizes around the chunks: 4 MiB exactly, a ragged last chunk, less
and more chunks than staging slots."""
import ctypes as C

import numpy as np
import pytest
import torch

import infinitempsalgorithms_b200 as imps
from infinitempsalgorithms_b200 import _lib as L

pytestmark = pytest.mark.gpu
PER_THREAD = 2   # cudaStreamPerThread


def _rc(rng, *s):
    return np.asfortranarray(rng.standard_normal(s) + 1j * rng.standard_normal(s))


@pytest.mark.parametrize("stream", ["own", "per_thread"])
@pytest.mark.parametrize("D,d", [(362, 2), (363, 2), (512, 1), (513, 3), (1024, 2)])
def test_round_trip(stream, D, d):
    ctx = imps.Context(0)
    if stream == "per_thread":
        L.check(ctx.lib.imps_ctx_set_stream(ctx.h, C.c_void_p(PER_THREAD)), ctx.h)
    rng = np.random.default_rng(D)
    psi = imps.CanonicalIMPS(ctx, [d], [D])
    for _ in range(3):
        A = _rc(rng, D, d, D)
        psi.set(L.IMPS_AC, 0, A)
        assert np.array_equal(psi.get(L.IMPS_AC, 0), A)
    del psi
    ctx.close()


@pytest.mark.parametrize("stream", ["own", "per_thread"])
def test_transfers_stay_behind_queued_applications(stream):
    D = 256
    ctx = imps.Context(0)
    if stream == "per_thread":
        L.check(ctx.lib.imps_ctx_set_stream(ctx.h, C.c_void_p(PER_THREAD)), ctx.h)
    H = imps.heisenberg_hamiltonian()
    m, d = H.Ws[0].shape[0], H.Ws[0].shape[1]
    rng = np.random.default_rng(1)
    psi = imps.CanonicalIMPS(ctx, [d], [D])
    envs = imps.DMRGCache(psi, H, build=False)
    GL, GL2, GR = (_rc(rng, D, m, D) / D for _ in range(3))
    assert GL.nbytes >= 4 << 20
    envs.set_leftenv(1, GL)
    envs.set_rightenv(1, GR)
    x = torch.from_numpy(np.ascontiguousarray(_rc(rng, D, d, D).T)).cuda()
    ys = [torch.empty_like(x) for _ in range(40)]
    torch.cuda.synchronize()

    def apply(y):
        L.check(ctx.lib.imps_ac_apply_dev(envs.h, H.handle(ctx), 0, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())),
                ctx.h)
    want = torch.empty_like(x)
    apply(want)
    ctx.synchronize()
    for y in ys:
        apply(y)
    envs.set_leftenv(1, GL2)   # behind the forty applications
    ctx.synchronize()
    assert all(torch.equal(y, want) for y in ys)
    M = _rc(rng, 1024, 512)    # an upload, a chain of kernels, downloads of their results
    Q, R = imps.qrpos(M, ctx=ctx)
    assert np.linalg.norm(Q @ R - M) <= 40 * np.sqrt(512) * np.finfo(float).eps * np.linalg.norm(M)
    del envs, psi
    ctx.close()
