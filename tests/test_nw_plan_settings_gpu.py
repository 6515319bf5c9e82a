"""Plans that a context keeps belong to the settings they were built under: a store's
calls before, during and after tiles that the caller sets."""
import ctypes

import numpy as np
import pytest
import torch

from msa_b200 import ScoringTable, _lib
from msa_b200 import workloads as W

pytestmark = pytest.mark.gpu

U8P, U64P = ctypes.POINTER(ctypes.c_uint8), ctypes.POINTER(ctypes.c_uint64)


def test_plans_of_fixed_tiles_are_not_taken_for_others(gpu):
    rng = np.random.default_rng(4)
    flat, offs, lens = W.Workload("plan", [W.DNA[rng.integers(0, 4, int(L))] for L in rng.integers(100, 250, 900)],
                                  "default", 0).flat_units()
    lib, t, n, h = _lib.lib(), ScoringTable("default"), len(lens), ctypes.c_uint64()
    _lib.check(lib.msa_seqs_upload(gpu.handle, flat.ctypes.data_as(U8P), offs.ctypes.data_as(U64P),
                                   lens.ctypes.data_as(U64P), n, ctypes.byref(h)), gpu.handle)
    out = torch.empty(n * (n - 1) // 2, dtype=torch.int32, device="cuda")

    def planes(tiles):
        _lib.check(lib.msa_nw_set_tiles(gpu.handle, *tiles))
        try:
            out.zero_()
            _lib.check(lib.msa_nw_all_pairs(gpu.handle, h.value, ctypes.byref(t._t), 0, ctypes.c_void_p(out.data_ptr()), 1),
                       gpu.handle)
            return lib.msa_nw_last_plane_tasks(gpu.handle), out.clone()
        finally:
            _lib.check(lib.msa_nw_set_tiles(gpu.handle, 0, 0))

    try:
        free, first = planes((0, 0))
        assert free > 0
        for tiles in ((32, 8), (0, 0), (32, 8), (0, 0)):   # 32 x 8 is also what the library chooses
            tasks, scores = planes(tiles)
            assert (tasks > 0) == (tiles == (0, 0))
            assert torch.equal(scores, first)
    finally:
        lib.msa_seqs_release(gpu.handle, h.value)
