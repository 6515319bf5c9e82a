"""Which calls run on bit planes, as msa_nw_last_plane_tasks reports it: the jobs whose
scores other tests compare are those that the path takes."""
import numpy as np
import pytest

from msa_b200 import ScoringTable, _lib, pairwise, runtime
from msa_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _planes(seqs, table, part=None, unclean=()):
    flat, offs, lens = W.Workload("route", seqs, "default", 0).flat_units()
    for k in unclean:
        flat[int(offs[k]) + 20: int(offs[k]) + 23] = 24
    if part is None:
        pairwise.score_units(flat, offs, lens, ScoringTable(table))
    else:
        pairwise.score_units_part(flat, offs, lens, ScoringTable(table), *part)
    return _lib.lib().msa_nw_last_plane_tasks(runtime.context(0).handle)


def _dna(rng, lens):
    return [W.DNA[rng.integers(0, 4, int(L))] for L in lens]


def test_jobs_on_bit_planes(gpu):
    rng = np.random.default_rng(1)
    reads = _dna(rng, rng.integers(100, 250, 900))
    assert _planes(reads, "default") > 0
    assert _planes(reads, "default", unclean=(3, 400, 899)) > 0
    for seed in (1, 2, 3):   # as test_nw_bits_gpu.test_uneven_lengths draws them
        r = np.random.default_rng(seed)
        assert _planes(_dna(rng, np.clip(np.exp(r.normal(6.5, 0.9, 700 + 37 * seed)), 1, 9000)), "default") > 0


def test_jobs_on_the_batched_kernel(gpu):
    rng = np.random.default_rng(2)
    reads = _dna(rng, rng.integers(100, 250, 900))
    assert _planes(reads, "blosum62") == 0
    assert _planes(reads[:32], "default") == 0
    assert _planes(reads, "default", part=(0, 2)) == 0
