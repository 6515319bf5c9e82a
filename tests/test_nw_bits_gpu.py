"""Pairs on bit planes (tables of one match and one mismatch score), at the edges
of their lanes, strips and column groups, against the oracle or, for the longer
ones, the plain kernel (one pair per warp, 32-bit lanes)."""
import numpy as np
import pytest

from msa_b200 import ScoringTable, _lib, pairwise, runtime
from msa_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


LETTERS = np.frombuffer(b"ACGTNX", np.uint8)   # X scores as a mismatch against itself


def _related(rng, lens, rate=0.3):
    """Sequences cut from one, each with its own substitutions and one deletion."""
    root = W.DNA[rng.integers(0, 4, int(max(lens)) + 40)]
    out = []
    for L in lens:
        at, k = (int(v) for v in rng.integers(0, (max(int(L) - 1, 1), 30)))
        s = np.concatenate([root[:at], root[at + k:]])[: int(L)].copy()
        m = rng.random(len(s)) < rate
        s[m] = LETTERS[rng.integers(0, 6, int(m.sum()))]
        out.append(s)
    return out


def _both(seqs, table):
    """Scores, the plain kernel's, and whether bit planes were used: their tasks
    are counted otherwise than the batched kernel's, which alone has tile shapes."""
    flat, offs, lens = W.Workload("bits", seqs, "default", 0).flat_units()
    ctx = runtime.context(0)
    got = pairwise.score_units(flat, offs, lens, table)
    tasks = pairwise.last_stats().narrow_tasks
    _lib.check(_lib.lib().msa_nw_set_tiles(ctx.handle, 32, 8))
    try:
        batched = pairwise.score_units(flat, offs, lens, table)
    finally:
        _lib.check(_lib.lib().msa_nw_set_tiles(ctx.handle, 0, 0))
    bits = tasks != pairwise.last_stats().narrow_tasks
    assert np.array_equal(got, batched)
    return got, pairwise.score_units(flat, offs, lens, table, _lib.MSA_NW_PLAIN), bits


# 8, 16 and 32 lanes per sequence (up to 256, 512 and more rows), one and several
# strips of 1,024 rows; counts that are and are not a multiple of 32 and of 4.
@pytest.mark.parametrize("n,lo,hi", [(2600, 20, 33), (2049, 31, 64), (1501, 60, 66), (1201, 120, 130), (800, 250, 262),
                                     (703, 505, 520), (512, 1000, 1030), (481, 1150, 1160), (333, 2040, 2060)])
def test_even_lengths(gpu, n, lo, hi):
    rng = np.random.default_rng(n)
    got, want, bits = _both(_related(rng, rng.integers(lo, hi + 1, n)), ScoringTable("default"))
    assert bits
    assert np.array_equal(got, want)


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_uneven_lengths(gpu, seed):
    """The longest sequences among themselves on the batched kernel, where that is quicker."""
    rng = np.random.default_rng(seed)
    lens = np.clip(np.exp(rng.normal(6.5, 0.9, 700 + 37 * seed)), 1, 9000)
    got, want, _ = _both(_related(rng, lens), ScoringTable("default"))
    assert np.array_equal(got, want)


def test_short_against_oracle(gpu, golden):
    rng = np.random.default_rng(7)
    seqs = _related(rng, rng.integers(36, 70, 1300))
    flat, offs, lens = W.Workload("bits", seqs, "default", 0).flat_units()
    got = pairwise.score_units(flat, offs, lens, ScoringTable("default"))
    want = O.oracle_nw_all_pairs(flat, offs, lens, O.table_block(golden), 7, O.TABLE_INDEX["default"], O.PENALTY["default"])
    assert np.array_equal(got, want)


def _table(match, mismatch, penalty, odd=None):
    s = np.full((25, 25), mismatch, np.int32)
    np.fill_diagonal(s, match)
    if odd:
        s[odd[0]] = odd[1]
    return ScoringTable.custom(s, penalty)


# u = 2 and 4; then tables that bit planes do not hold: another ratio, one entry
# that differs, no gap penalty, u = 0.
@pytest.mark.parametrize("table,bits", [
    (_table(2, -2, 2), True), (_table(4, -4, 4), True), (_table(5, -1, 1), False),
    (_table(1, -1, 1, ((3, 1), 0)), False), (_table(3, 1, 0), True), (_table(1, -2, 1), False)])
def test_other_tables(gpu, table, bits):
    rng = np.random.default_rng(11)
    got, want, used = _both(_related(rng, rng.integers(90, 200, 1000)), table)
    assert used == bits
    assert np.array_equal(got, want)


def test_unclean_sequences(gpu):
    """END units inside some sequences: their pairs on the other kernel, the rest on bit planes."""
    rng = np.random.default_rng(12)
    flat, offs, lens = W.Workload("bits", _related(rng, rng.integers(100, 250, 900)), "default", 0).flat_units()
    for k in (3, 400, 899):
        flat[int(offs[k]) + 20: int(offs[k]) + 23] = 24
    got = pairwise.score_units(flat, offs, lens, ScoringTable("default"))
    assert np.array_equal(got, pairwise.score_units(flat, offs, lens, ScoringTable("default"), _lib.MSA_NW_PLAIN))
