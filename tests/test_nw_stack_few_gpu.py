"""Jobs of 95 to 190 sequences, where rows pairs are stacked two by two if their tasks
are alike and more than the chip holds at once, against the plain kernel."""
import numpy as np
import pytest

from msa_b200 import ScoringTable, _lib, pairwise
from msa_b200 import workloads as W

pytestmark = pytest.mark.gpu


# Around the number of tasks from which on they are stacked, up to that at which they
# always are; alike, of two kinds, and up to past the 512 rows of a stacked pair.
@pytest.mark.parametrize("n", [90, 93, 94, 100, 151, 189, 190])
@pytest.mark.parametrize("lo,hi", [(1, 4), (20, 30), (250, 258), (480, 512), (500, 520), (40, 500)])
def test_few_short_sequences_match(gpu, n, lo, hi):
    rng = np.random.default_rng(n * hi)
    root = W.AMINO[rng.integers(0, 20, hi)]
    seqs = []
    for L in rng.integers(lo, hi + 1, n):
        s = root[: int(L)].copy()
        m = rng.random(len(s)) < 0.2
        s[m] = W.AMINO[rng.integers(0, 20, int(m.sum()))]
        seqs.append(s)
    flat, offs, lens = W.Workload("few", seqs, "blosum62", 0).flat_units()
    table = ScoringTable("blosum62")
    assert np.array_equal(pairwise.score_units(flat, offs, lens, table),
                          pairwise.score_units(flat, offs, lens, table, _lib.MSA_NW_PLAIN))
