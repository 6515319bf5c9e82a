"""Rows pairs of several strips on 16-bit lanes with a moving base, chained over
the CTAs or not, against the oracle and the 32-bit lanes."""
import numpy as np
import pytest

from msa_b200 import ScoringTable, _lib, pairwise, runtime
from msa_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _score(wl, table, variant=0):
    ctx = runtime.context(0)
    flat, offs, lens = wl.flat_units()
    _lib.check(_lib.lib().msa_nw_set_variant(ctx.handle, variant, 0))
    try:
        return pairwise.score_units(flat, offs, lens, table)
    finally:
        _lib.check(_lib.lib().msa_nw_set_variant(ctx.handle, 0, 0))


def _related(rng, lens, alphabet, rate):
    """Sequences cut from one, each with its own substitutions: scores far from zero."""
    root = alphabet[rng.integers(0, len(alphabet), max(lens) + 50)]
    out = []
    for L in lens:
        s = root[: int(L)].copy()
        m = rng.random(len(s)) < rate
        s[m] = alphabet[rng.integers(0, len(alphabet), int(m.sum()))]
        out.append(s)
    return out


# Lengths at the edges of strips (1,024 rows, or 512 and 256 where they are
# lowered), of the base's moves (512 columns) and of 32-column blocks; values
# that pass 16 bits (blosum62: 19 per match, from 3,450 residues on).
@pytest.mark.parametrize("lens,table", [
    ([1025, 1024, 1023], "default"), ([1055, 1056, 1057, 31, 32, 33], "blosum62"),
    ([2048, 2049, 2047, 512, 481, 480, 513], "blosum62"), ([3600, 3599, 3450, 3449, 1], "blosum62"),
    ([7000, 6900, 5000, 4097, 4096, 900, 17], "blosum62"), ([5200, 5100, 300], "pam250"),
    ([22000, 21900, 9000], "default"), ([1500] * 20, "blosum45"),
])
def test_long_rows_match_oracle(gpu, golden, lens, table):
    rng = np.random.default_rng(sum(lens))
    alphabet = W.DNA if table == "default" else W.AMINO
    wl = W.Workload("long", _related(rng, lens, alphabet, 0.1), table, 0)
    t = ScoringTable(table)
    got = _score(wl, t)
    if len(lens) < 8:
        flat, offs, lens3 = wl.flat_units()
        want = O.oracle_nw_all_pairs(flat, offs, lens3, O.table_block(golden), 7, O.TABLE_INDEX[table], O.PENALTY[table])
        assert np.array_equal(got, want)
    assert np.array_equal(got, _score(wl, t, _lib.MSA_NW_VARIANT_INT32))


def test_many_long_rows_unchained(gpu):
    """Enough long rows pairs that none is chained: the moving base over all
    strips of a task."""
    rng = np.random.default_rng(5)
    lens = rng.integers(3500, 3900, 160)
    wl = W.Workload("long", _related(rng, lens, W.AMINO, 0.3), "blosum62", 0)
    t = ScoringTable("blosum62")
    assert np.array_equal(_score(wl, t), _score(wl, t, _lib.MSA_NW_VARIANT_INT32))
