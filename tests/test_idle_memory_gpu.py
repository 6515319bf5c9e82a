"""Device memory that a context keeps for later calls (plans, blocks of released
stores) is given back when the caller asks, and when an allocation of the context finds
none left."""
import ctypes

import numpy as np
import pytest
import torch

from msa_b200 import ScoringTable, _lib, runtime
from msa_b200 import workloads as W

pytestmark = pytest.mark.gpu

U8P, U64P = ctypes.POINTER(ctypes.c_uint8), ctypes.POINTER(ctypes.c_uint64)
MB = 1 << 20


def _upload(ctx, flat, offs, lens):
    h = ctypes.c_uint64()
    _lib.check(_lib.lib().msa_seqs_upload(ctx.handle, flat.ctypes.data_as(U8P), offs.ctypes.data_as(U64P),
                                          lens.ctypes.data_as(U64P), len(lens), ctypes.byref(h)), ctx.handle)
    return h.value


def _leave_free(ctx, mb, blocks):
    """Releases two stores of `blocks` MB, which the context keeps, then fills the
    device but for `mb` MB."""
    flat = np.zeros(blocks * MB, np.uint8)
    one = np.array([len(flat)], np.uint64)
    handles = [_upload(ctx, flat, np.zeros(1, np.uint64), one) for _ in range(2)]
    before = torch.cuda.mem_get_info()[0]
    for h in handles:
        _lib.check(_lib.lib().msa_seqs_release(ctx.handle, h))
    assert torch.cuda.mem_get_info()[0] - before < blocks * MB   # kept, not freed
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - mb * MB, dtype=torch.uint8, device="cuda")


@pytest.fixture
def ctx(gpu):
    torch.cuda.empty_cache()
    c = runtime.Context(0)
    yield c
    c.close()
    torch.cuda.empty_cache()


def test_plans_and_blocks_are_released_on_request(ctx):
    rng = np.random.default_rng(1)
    flat, offs, lens = W.Workload("idle", [W.AMINO[rng.integers(0, 20, 3000)] for _ in range(60)], "blosum62", 0).flat_units()
    t, out = ScoringTable("blosum62"), torch.empty(60 * 59 // 2, dtype=torch.int32, device="cuda")
    h = _upload(ctx, flat, offs, lens)

    def score():
        out.zero_()
        _lib.check(_lib.lib().msa_nw_all_pairs(ctx.handle, h, ctypes.byref(t._t), 0, ctypes.c_void_p(out.data_ptr()), 1),
                   ctx.handle)
        return out.clone()

    first = score()
    before = torch.cuda.mem_get_info()[0]
    _lib.check(_lib.lib().msa_release_idle(ctx.handle))
    assert torch.cuda.mem_get_info()[0] - before >= 4 * MB   # the plan's profiles alone: 26 B per residue
    assert torch.equal(score(), first)
    assert torch.equal(score(), first)
    _lib.check(_lib.lib().msa_seqs_release(ctx.handle, h))


def test_a_tree_takes_the_memory_of_idle_blocks(ctx):
    n = 9000   # its matrix and the next stage's take 440 MB
    tri = torch.from_numpy(np.random.default_rng(2).integers(50, 400, n * (n - 1) // 2).astype(np.int32)).cuda()
    nodes = (_lib.MsaOtu * (2 * n - 1))()

    def tree():
        _lib.check(_lib.lib().msa_nj_order(ctx.handle, ctypes.c_void_p(tri.data_ptr()), _lib.MSA_TRI_I32_DEVICE, n,
                                           _lib.MSA_NJ_SYMMETRIC, nodes), ctx.handle)
        return bytes(nodes)

    fill = _leave_free(ctx, 200, 400)
    got = tree()
    del fill
    torch.cuda.empty_cache()
    assert got == tree()


def test_scores_take_the_memory_of_idle_blocks(ctx):
    n = 9000   # 162 MB of scores, copied to the host through a buffer of the context
    rng = np.random.default_rng(3)
    flat, offs, lens = W.Workload("idle", [W.DNA[rng.integers(0, 4, 30)] for _ in range(n)], "default", 0).flat_units()
    t = ScoringTable("default")
    out = np.zeros(n * (n - 1) // 2, np.int32)
    h = _upload(ctx, flat, offs, lens)
    fill = _leave_free(ctx, 64, 400)
    _lib.check(_lib.lib().msa_nw_all_pairs(ctx.handle, h, ctypes.byref(t._t), 0, out.ctypes.data_as(ctypes.c_void_p), 0),
               ctx.handle)
    del fill
    assert out[-1] == _pair_score(flat, offs, lens, n - 1, n - 2)
    _lib.check(_lib.lib().msa_seqs_release(ctx.handle, h))


def test_ties_without_memory_for_the_packed_matrix(ctx):
    """A launch that gives up finds no memory for the other kernel's matrix: the tree is
    built without giving up."""
    n = 3000
    tri = np.full(n * (n - 1) // 2, 500, np.float32)
    nodes = (_lib.MsaOtu * (2 * n - 1))()

    def tree():
        _lib.check(_lib.lib().msa_nj_order(ctx.handle, tri.ctypes.data_as(ctypes.c_void_p), _lib.MSA_TRI_F32_HOST, n,
                                           _lib.MSA_NJ_SYMMETRIC, nodes), ctx.handle)
        return bytes(nodes)

    want = tree()
    _lib.check(_lib.lib().msa_release_idle(ctx.handle))
    free = torch.cuda.mem_get_info()[0]
    fill = torch.empty(free - 16 * MB, dtype=torch.uint8, device="cuda")
    assert tree() == want
    del fill


def _pair_score(flat, offs, lens, i, j):
    """Needleman-Wunsch score of one pair by the definition (match 1, mismatch -1, gap 1)."""
    a, b = (flat[int(offs[k]): int(offs[k]) + int(lens[k])] for k in (i, j))
    a, b = a[a < 24], b[b < 24]
    row = -np.arange(len(b) + 1)
    for x in a:
        new = np.empty_like(row)
        new[0] = row[0] - 1
        for q in range(len(b)):
            new[q + 1] = max(row[q] + (1 if x == b[q] else -1), row[q + 1] - 1, new[q] - 1)
        row = new
    return int(row[-1])
