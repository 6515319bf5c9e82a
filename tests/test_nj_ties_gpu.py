"""Matrices in which many pairs tie (copies of a sequence, few distinct scores),
where the joining kernel's launches give up and the kernel that searches every
pair takes over: the same trees as the oracle's, and no more than a few times the
time of a matrix without ties."""
import time

import numpy as np
import pytest

from msa_b200 import _lib, phylogeny
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _matrix(n, kind, rng):
    i, j = np.tril_indices(n, -1)
    if kind == "equal":
        return np.full(len(i), 500, np.float32)
    if kind == "outbreak":   # a few mutations each; row sums beyond 2^24 from 600 nodes on
        m = rng.poisson(3, n)
        return (29900 - 2 * (m[i] + m[j])).astype(np.float32)
    if kind == "huge":       # the bounds are off, nearly every Q is rounded to the same value
        tri = np.round(rng.normal(100, 40, len(i))).astype(np.float32)
        tri[rng.integers(0, len(i), 3)] = 1e30
        return tri
    if kind.startswith("late"):   # copies of one that join after that many others have
        k = int(kind[4:])
        ids = rng.permutation(n)
        x = np.round(rng.normal(0, 300, (n, 4)))
        a, b = ids[i] < k, ids[j] < k
        d = 3000 - np.abs(x[ids[i]] - x[ids[j]]).sum(-1)
        return np.where(a & b, d, np.where(a | b, 100, 1000)).astype(np.float32)
    if kind == "scores":
        return np.round(rng.normal(100, 40, len(i))).astype(np.float32)
    # Copies of `kind` distinct sequences, or of one among as many others.
    ids = rng.integers(0, int(kind), n) if int(kind) < n // 2 else np.maximum(np.arange(n) - int(kind), 0)
    rng.shuffle(ids)
    x = np.round(rng.normal(0, 60, (ids.max() + 1, 6)))
    return (800 - np.abs(x[ids[i]] - x[ids[j]]).sum(-1)).astype(np.float32)


# Sizes whose launches never give up, that do so after a few joins, in the first,
# second and third launch (the matrix and the row sums change places), at sizes at
# the edges of a chunk and of a batch of loads.
@pytest.mark.parametrize("order", ["symmetric", "linear"])
@pytest.mark.parametrize("n,kind", [(231, "equal"), (385, "equal"), (513, "huge"), (700, "outbreak"), (1201, "outbreak"),
                                    (1030, "7"), (777, "40"), (900, "450"), (1500, "900"), (640, "huge"),
                                    (1500, "late750"), (1500, "late1050")])
def test_ties_match_oracle(gpu, n, kind, order):
    tri = _matrix(n, kind, np.random.default_rng(n))
    got = phylogeny.run_triangle(tri, n, order=_lib.MSA_NJ_LINEAR if order == "linear" else _lib.MSA_NJ_SYMMETRIC)
    want = O.oracle_nj(tri, n, order)
    for k in ("parent", "child0", "child1", "level"):
        assert np.array_equal(np.asarray(getattr(got, k)), np.asarray(want[k]))
    assert np.array_equal(got.distance.view(np.uint32), np.asarray(want["distance"], np.float32).view(np.uint32))


def _seconds(tri, n):
    best = np.inf
    for _ in range(4):
        start = time.perf_counter()
        phylogeny.run_triangle(tri, n)
        best = min(best, time.perf_counter() - start)
    return best


@pytest.mark.parametrize("kind", ["equal", "outbreak", "7", "1000"])
def test_ties_cost_no_more_than_a_search_of_every_pair(gpu, kind):
    """A search of all pairs at every join takes twice the bounded one's time at
    this size; one that goes through tied cells again took it to 17 times."""
    n = 2000
    rng = np.random.default_rng(1)
    assert _seconds(_matrix(n, kind, rng), n) < 4 * _seconds(_matrix(n, "scores", rng), n)
