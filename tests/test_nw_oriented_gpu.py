"""Inputs whose scores depend on the orientation of a pair (GAP units, tables
that are not symmetric) on the batched and plain kernels, which take them in the
reference's orientation as one sorted order, against the oracle."""
import ctypes

import numpy as np
import pytest

from msa_b200 import ScoringTable, _lib, pairwise
from msa_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _set(seed, n, lo, hi, gaps=0.05, suffix=0, inside=0):
    """Proteins with '-' runs; `suffix` of them end in up to 7 END characters
    (whole blocks of them in some), `inside` of them hold END units inside."""
    rng = np.random.default_rng(seed)
    seqs = []
    for k in range(n):
        s = W.AMINO[rng.integers(0, 20, int(rng.integers(lo, hi + 1)))].copy()
        if k % 5:
            s[rng.random(len(s)) < gaps] = ord("-")
        if k < suffix:
            s = np.concatenate([s, np.full(int(rng.integers(1, 8)), ord("*"), np.uint8)])
        elif k < suffix + inside:
            s[len(s) // 2] = ord("*")
        seqs.append(s)
    order = rng.permutation(n)
    return W.Workload("oriented", [seqs[k] for k in order], "blosum62", seed)


def _asymmetric(rng, spread, penalty):
    return ScoringTable.custom(rng.integers(-spread, spread + 1, 625), penalty), penalty


def _check(wl, table, tables, count, index, penalty):
    flat, offs, lens = wl.flat_units()
    want = O.oracle_nw_all_pairs(flat, offs, lens, tables, count, index, penalty)
    for mode in (_lib.MSA_NW_PERSISTENT, _lib.MSA_NW_PLAIN):
        assert np.array_equal(pairwise.score_units(flat, offs, lens, table, mode), want)
    total = np.zeros_like(want)
    for part in range(3):
        total += pairwise.score_units_part(flat, offs, lens, table, part, 3)
    assert np.array_equal(total, want)


# Few distinct block counts, so that ties decide; one strip, several, stacked
# rows pairs (from 275 sequences on) and chained strips.
@pytest.mark.parametrize("n,lo,hi,suffix,inside", [(2, 3, 9, 0, 0), (33, 1, 12, 0, 0), (40, 95, 104, 9, 3),
                                                   (300, 20, 40, 0, 0), (290, 120, 300, 0, 1), (12, 1000, 1100, 2, 1),
                                                   (7, 2400, 2500, 1, 0)])
@pytest.mark.parametrize("name", ["blosum62", "blosum45"])
def test_gap_units_match_oracle(gpu, golden, name, n, lo, hi, suffix, inside):
    _check(_set(n + hi, n, lo, hi, suffix=suffix, inside=inside), ScoringTable(name), O.table_block(golden), 7,
           O.TABLE_INDEX[name], O.PENALTY[name])


@pytest.mark.parametrize("n,lo,hi,spread,penalty", [(21, 1, 20, 4, 3), (300, 15, 35, 4, 3), (30, 200, 260, 9, 2),
                                                    (6, 1500, 1600, 5, 4), (10, 100, 400, 127, 90)])
def test_asymmetric_tables_match_oracle(gpu, n, lo, hi, spread, penalty):
    rng = np.random.default_rng(n + lo)
    table, penalty = _asymmetric(rng, spread, penalty)
    m = table.matrix()
    _check(_set(n, n, lo, hi, gaps=0.0, suffix=n // 4, inside=n // 10), table, np.ascontiguousarray(m.reshape(-1)), 1, 0,
           penalty)


def test_one_store_under_both_orders(gpu, golden):
    """A symmetric, then an asymmetric, then a symmetric table on one store:
    each call uses its own order."""
    wl = _set(9, 30, 60, 90, gaps=0.0)
    flat, offs, lens = wl.flat_units()
    rng = np.random.default_rng(3)
    table, penalty = _asymmetric(rng, 6, 4)
    u8, u64 = ctypes.POINTER(ctypes.c_uint8), ctypes.POINTER(ctypes.c_uint64)
    h = ctypes.c_uint64()
    lib = _lib.lib()
    _lib.check(lib.msa_seqs_upload(gpu.handle, flat.ctypes.data_as(u8), offs.ctypes.data_as(u64),
                                   lens.ctypes.data_as(u64), len(lens), ctypes.byref(h)), gpu.handle)
    try:
        sym = O.oracle_nw_all_pairs(flat, offs, lens, O.table_block(golden), 7, O.TABLE_INDEX["pam250"], O.PENALTY["pam250"])
        asym = O.oracle_nw_all_pairs(flat, offs, lens, np.ascontiguousarray(table.matrix().reshape(-1)), 1, 0, penalty)
        for t, want in ((ScoringTable("pam250"), sym), (table, asym), (ScoringTable("pam250"), sym), (table, asym)):
            out = np.zeros(len(want), np.int32)
            _lib.check(lib.msa_nw_all_pairs(gpu.handle, h.value, ctypes.byref(t._t), 0,
                                            out.ctypes.data_as(ctypes.c_void_p), 0), gpu.handle)
            assert np.array_equal(out, want)
    finally:
        lib.msa_seqs_release(gpu.handle, h.value)
