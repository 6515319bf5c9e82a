"""Trees of different sizes built at once by threads with contexts of their own, which
launch the same kernels with different amounts of shared memory."""
import ctypes
import threading

import numpy as np
import pytest

from msa_b200 import _lib, runtime

pytestmark = pytest.mark.gpu


def _tree(ctx, tri, n):
    nodes = (_lib.MsaOtu * (2 * n - 1))()
    _lib.check(_lib.lib().msa_nj_order(ctx.handle, tri.ctypes.data_as(ctypes.c_void_p), _lib.MSA_TRI_F32_HOST, n,
                                       _lib.MSA_NJ_SYMMETRIC, nodes), ctx.handle)
    return bytes(nodes)


# One CTA of 16 warps; one cluster (then one CTA again).
@pytest.mark.parametrize("sizes", [(70, 229, 120, 200), (240, 1500, 260, 900)])
def test_threads_with_different_sizes(gpu, sizes):
    rng = np.random.default_rng(sizes[0])
    tris = [np.round(rng.normal(100, 40, n * (n - 1) // 2)).astype(np.float32) for n in sizes]
    want = [_tree(gpu, t, n) for t, n in zip(tris, sizes)]
    wrong = []

    def work(k):
        try:
            ctx = runtime.Context(0)
            for _ in range(300 if sizes[k] < 230 else 100):
                if _tree(ctx, tris[k], sizes[k]) != want[k]:
                    wrong.append((sizes[k], "another tree"))
            ctx.close()
        except Exception as e:
            wrong.append((sizes[k], repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
