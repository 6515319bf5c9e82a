"""Matrices whose Q values do not fit 24 bits, with many near ties: a product that is
not rounded before the row sums are subtracted takes other joins."""
import numpy as np
import pytest

from msa_b200 import _lib, phylogeny, runtime
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _matrix(n, kind):
    rng = np.random.default_rng(n)
    i, j = np.tril_indices(n, -1)
    if kind == "outbreak":   # genomes of one length with a few mutations each
        m = rng.poisson(5, n)
        return (29900 - 2 * (m[i] + m[j])).astype(np.float32)
    tri = np.round(rng.normal(100, 40, len(i))).astype(np.float32)
    tri[rng.integers(0, len(i), 3)] = 1e30
    return tri


@pytest.mark.parametrize("order", ["symmetric", "linear"])
@pytest.mark.parametrize("n,kind", [(1200, "outbreak"), (700, "huge")])
@pytest.mark.parametrize("clusters", [0, 2, 4])
def test_rounded_products_match_oracle(gpu, n, kind, order, clusters):
    tri = _matrix(n, kind)
    ctx = runtime.context(0)
    _lib.check(_lib.lib().msa_nj_set_clusters(ctx.handle, clusters, 8, 0, 0))
    try:
        got = phylogeny.run_triangle(tri, n, order=_lib.MSA_NJ_LINEAR if order == "linear" else _lib.MSA_NJ_SYMMETRIC)
    finally:
        _lib.check(_lib.lib().msa_nj_set_clusters(ctx.handle, 0, 0, 0, 0))
    want = O.oracle_nj(tri, n, order)
    for k in ("parent", "child0", "child1", "level"):
        assert np.array_equal(np.asarray(getattr(got, k)), np.asarray(want[k]))
    assert np.array_equal(got.distance.view(np.uint32), np.asarray(want["distance"], np.float32).view(np.uint32))
