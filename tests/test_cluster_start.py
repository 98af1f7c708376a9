"""A CTA may touch a peer's shared memory only once that peer runs, so a kernel that stores into
its cluster has a cluster barrier before its first remote access.  Read from the sources; the
row counts where whole CTAs of the QR panel's cluster own no rows are run on the device."""
import re
from pathlib import Path

import numpy as np
import pytest

import infinitempsalgorithms_b200 as imps

CSRC = Path(imps.__file__).parent / "csrc"
REMOTE = re.compile(r"\bst_peer\(|\bpublish\(|\bleader_addr\(|shared::cluster\.(?:v2\.)?f64 ")
BARRIER = re.compile(r"\bcluster_wait\(\)|\bcluster_sync\(\)|barrier\.cluster\.wait")


def _cluster_kernels():
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        for m in re.finditer(r"__cluster_dims__\([^)]*\)[^{;]*?\b(k_\w+)\([^{;]*\{", text):
            end = text.index("\n}\n", m.end())
            yield path.name, m.group(1), text[m.end():end]


KERNELS = list(_cluster_kernels())


def test_the_cluster_kernels_are_found():
    assert {"k_qr_panel", "k_ac_small", "k_mod_gemm"} <= {k for _, k, _ in KERNELS}


@pytest.mark.parametrize("name,kernel,body", KERNELS, ids=[k for _, k, _ in KERNELS])
def test_a_cluster_barrier_precedes_the_first_remote_access(name, kernel, body):
    first = REMOTE.search(body)
    assert first, "a cluster kernel without remote accesses"
    barrier = BARRIER.search(body)
    assert barrier and barrier.start() < first.start()


@pytest.mark.gpu
@pytest.mark.parametrize("m", [257, 260, 320, 513, 1025, 2049])
def test_panels_whose_last_ctas_own_no_rows(m):
    """Backward error of Householder QR, and the same bits every time."""
    rng = np.random.default_rng(m)
    n = 16
    M = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    ctx = imps.Context(0)
    Q0, R0 = imps.qrpos(M, ctx=ctx)
    assert np.linalg.norm(Q0 @ R0 - M) <= 40 * np.sqrt(n) * np.finfo(float).eps * np.linalg.norm(M)
    for _ in range(20):
        Q, R = imps.qrpos(M, ctx=ctx)
        assert np.array_equal(Q, Q0) and np.array_equal(R, R0)
    ctx.close()
