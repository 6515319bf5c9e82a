"""Waits between the strips of a long sequence that run out (a limit of 1 us, less than
a strip takes for the first columns that the next one waits for): the call fails with
a status, and the next call on the same store and context scores it."""
import ctypes

import numpy as np
import pytest

from msa_b200 import ScoringTable, _lib, pairwise, runtime
from msa_b200 import workloads as W

pytestmark = pytest.mark.gpu

U8P, U64P = ctypes.POINTER(ctypes.c_uint8), ctypes.POINTER(ctypes.c_uint64)


# Strips over several CTAs on 16-bit lanes, of proteins and of DNA; over the warps of
# a CTA on bit planes.
@pytest.mark.parametrize("lens,table", [([5000] * 6, "blosum62"), ([9000] * 3 + [3000] * 40, "default"),
                                        ([12000] + [400] * 1500, "default")])
def test_waits_run_out_and_the_context_stays_usable(gpu, lens, table):
    rng = np.random.default_rng(len(lens))
    alphabet = W.DNA if table == "default" else W.AMINO
    seqs = [alphabet[rng.integers(0, len(alphabet), L)] for L in lens]
    flat, offs, lens3 = W.Workload("wait", seqs, table, 0).flat_units()
    t, lib, n = ScoringTable(table), _lib.lib(), len(lens)
    want = pairwise.score_units(flat, offs, lens3, t, _lib.MSA_NW_PLAIN)
    h = ctypes.c_uint64()
    _lib.check(lib.msa_seqs_upload(gpu.handle, flat.ctypes.data_as(U8P), offs.ctypes.data_as(U64P),
                                   lens3.ctypes.data_as(U64P), n, ctypes.byref(h)), gpu.handle)
    out = np.zeros(n * (n - 1) // 2, np.int32)

    def score():
        return lib.msa_nw_all_pairs(gpu.handle, h.value, ctypes.byref(t._t), 0, out.ctypes.data_as(ctypes.c_void_p), 0)

    try:
        _lib.check(score(), gpu.handle)   # the plan that the failing call must not damage
        for _ in range(2):
            _lib.check(lib.msa_nw_set_wait(gpu.handle, 1))
            try:
                assert score() == _lib.MSA_ERR_DEVICE_TIMEOUT
                assert score() == _lib.MSA_ERR_DEVICE_TIMEOUT   # its kept plan
            finally:
                _lib.check(lib.msa_nw_set_wait(gpu.handle, 0))
            out[:] = 0
            _lib.check(score(), gpu.handle)
            assert np.array_equal(out, want)
    finally:
        lib.msa_seqs_release(gpu.handle, h.value)
