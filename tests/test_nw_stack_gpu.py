"""Short rows pairs stacked two and four to a warp, at the edges of their lanes
(8 and 16 lanes of up to 32 rows), against the oracle, or for the longer ones
against the plain kernel (one pair per warp, 32-bit lanes)."""
import numpy as np
import pytest

from msa_b200 import ScoringTable, _lib, pairwise
from msa_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# 275 sequences and more give enough tasks to be stacked; an odd count leaves a
# rows pair of one sequence, and counts that are not a multiple of 8 a rest.
@pytest.mark.parametrize("n,lo,hi", [(280, 1, 3), (283, 1, 17), (277, 30, 66), (276, 254, 258), (281, 60, 256),
                                     (276, 505, 518), (290, 1, 520)])
@pytest.mark.parametrize("table", ["blosum62", "default"])
def test_stacked_rows_pairs_match(gpu, golden, n, lo, hi, table):
    rng = np.random.default_rng(n + hi)
    alphabet = W.DNA if table == "default" else W.AMINO
    root = alphabet[rng.integers(0, len(alphabet), hi)]
    seqs = []
    for L in rng.integers(lo, hi + 1, n):
        s = root[: int(L)].copy()
        m = rng.random(len(s)) < 0.2
        s[m] = alphabet[rng.integers(0, len(alphabet), int(m.sum()))]
        seqs.append(s)
    flat, offs, lens = W.Workload("stack", seqs, table, 0).flat_units()
    if hi < 100:
        want = O.oracle_nw_all_pairs(flat, offs, lens, O.table_block(golden), 7, O.TABLE_INDEX[table], O.PENALTY[table])
    else:
        want = pairwise.score_units(flat, offs, lens, ScoringTable(table), _lib.MSA_NW_PLAIN)
    assert np.array_equal(pairwise.score_units(flat, offs, lens, ScoringTable(table)), want)
