"""Rows pairs in the reference's orientation whose two sequences have the same number
of 3-unit blocks but lie on both sides of a multiple of 1,024 rows, where the first
one's score profile ends before the strips do."""
import numpy as np
import pytest

from msa_b200 import ScoringTable, _lib, pairwise
from msa_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _set(lens, seed):
    rng = np.random.default_rng(seed)
    root = W.AMINO[rng.integers(0, 20, max(lens))]
    seqs = []
    for L in lens:   # related, so that scores come near the largest of their length; '-' in all
        s = root[:L].copy()
        m = rng.random(L) < 0.1
        s[m] = W.AMINO[rng.integers(0, 20, int(m.sum()))]
        s[rng.random(L) < 0.03] = ord("-")
        seqs.append(s)
    return W.Workload("edge", seqs, "blosum62", 0)


# The shorter one first and last in the store and in its rows pair; chained strips
# (few sequences), strips one after the other (many), and a moving base.
@pytest.mark.parametrize("lens", [[1024, 1026], [1026, 1024], [1025, 1024, 1026, 1024], [1024, 1024, 1025, 1026, 900],
                                  [2048, 2049, 2047], [2049, 2048, 2047, 2048], [4096, 4098, 4097, 4096],
                                  [1024, 1025, 1026] * 37, [2048, 2049, 2047] * 25])
def test_profiles_that_end_within_a_strip(gpu, golden, lens):
    wl = _set(lens, sum(lens))
    flat, offs, lens3 = wl.flat_units()
    table = ScoringTable("blosum62")
    got = pairwise.score_units(flat, offs, lens3, table)
    if len(lens) < 8:
        assert np.array_equal(got, O.oracle_nw_all_pairs(flat, offs, lens3, O.table_block(golden), 7,
                                                         O.TABLE_INDEX["blosum62"], O.PENALTY["blosum62"]))
    assert np.array_equal(got, pairwise.score_units(flat, offs, lens3, table, _lib.MSA_NW_PLAIN))
