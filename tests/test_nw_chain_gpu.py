"""Jobs of long rows pairs: which of them are chained over the CTAs (strips as tasks that
follow one another) and with which strips, at sizes on both sides of the rule, against
the plain kernel; and the time of jobs that chaining made slower."""
import ctypes
import time

import numpy as np
import pytest
import torch

from msa_b200 import ScoringTable, _lib, pairwise
from msa_b200 import workloads as W

pytestmark = pytest.mark.gpu

U8P, U64P = ctypes.POINTER(ctypes.c_uint8), ctypes.POINTER(ctypes.c_uint64)


def _units(lens, seed):
    rng = np.random.default_rng(seed)
    root = W.AMINO[rng.integers(0, 20, max(lens))]
    seqs = []
    for L in lens:
        s = root[:L].copy()
        m = rng.random(L) < 0.3
        s[m] = W.AMINO[rng.integers(0, 20, int(m.sum()))]
        seqs.append(s)
    return W.Workload("chain", seqs, "blosum62", 0).flat_units()


# Strips of up to 1,024 rows, of 512, and none chained; one long sequence among short ones.
@pytest.mark.parametrize("lens", [[1030] * 8, [1500] * 6, [1500, 1490] * 20, [1030] * 50, [2100] * 17, [2100] * 50,
                                  [3000] * 5, [4200, 4100, 4000], [1030] * 130, [9000] + [200] * 40,
                                  [9000] + [150] * 300, [1500] + [100] * 33, [5000, 3000, 1100] + [300] * 60])
def test_forms_of_long_rows_pairs(gpu, lens):
    flat, offs, lens3 = _units(lens, len(lens) + lens[0])
    table = ScoringTable("blosum62")
    assert np.array_equal(pairwise.score_units(flat, offs, lens3, table),
                          pairwise.score_units(flat, offs, lens3, table, _lib.MSA_NW_PLAIN))


def _seconds(ctx, lens):
    flat, offs, lens3 = _units(lens, 5)
    t, lib, n = ScoringTable("blosum62"), _lib.lib(), len(lens)
    out, h, best = torch.empty(n * (n - 1) // 2, dtype=torch.int32, device="cuda"), ctypes.c_uint64(), np.inf
    try:
        _lib.check(lib.msa_seqs_upload(ctx.handle, flat.ctypes.data_as(U8P), offs.ctypes.data_as(U64P),
                                       lens3.ctypes.data_as(U64P), n, ctypes.byref(h)), ctx.handle)
        for _ in range(5):
            start = time.perf_counter()
            _lib.check(lib.msa_nw_all_pairs(ctx.handle, h.value, ctypes.byref(t._t), 0, ctypes.c_void_p(out.data_ptr()), 1),
                       ctx.handle)
            best = min(best, time.perf_counter() - start)
    finally:
        lib.msa_seqs_release(ctx.handle, h.value)
    return best


def _unchained_seconds(ctx, lens):
    """Tiles that the caller sets keep every strip of a rows pair in one task."""
    _lib.check(_lib.lib().msa_nw_set_tiles(ctx.handle, 32, 8))
    try:
        return _seconds(ctx, lens)
    finally:
        _lib.check(_lib.lib().msa_nw_set_tiles(ctx.handle, 0, 0))


@pytest.mark.parametrize("lens", [[1030] * 64, [1500] * 64, [20000] + [200] * 49, [20000] + [200] * 699])
def test_chaining_is_not_slower(gpu, lens):
    """These took 1.5 to 2.5 times as long chained."""
    assert _seconds(gpu, lens) < 1.25 * _unchained_seconds(gpu, lens)
