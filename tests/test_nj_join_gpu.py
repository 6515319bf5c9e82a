"""The joining kernels of neighbor-joining at the sizes where their launches
change (one CTA of four or sixteen warps, one cluster, packed in stages) and on
matrices that their bounds and their split row-sum fold find hard, against the
oracle, or, where the reference's NaN arithmetic decides, against the kernel
that scans every pair."""
import numpy as np
import pytest

from msa_b200 import _lib, phylogeny, runtime
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _same(got, want):
    for k in ("parent", "child0", "child1", "level"):
        assert np.array_equal(np.asarray(getattr(got, k)), np.asarray(want[k]))
    assert np.array_equal(got.distance.view(np.uint32), np.asarray(want["distance"], np.float32).view(np.uint32))


def _matrix(n, kind, rng):
    m = n * (n - 1) // 2
    if kind == "scores":     # integers of one sign: long runs of one binade in the fold
        return np.round(rng.normal(-300, 40, m)).astype(np.float32)
    if kind == "balanced":   # row sums that keep crossing zero
        return (rng.integers(0, 2, m) * 2 - 1).astype(np.float32) * rng.integers(1, 2000, m)
    if kind == "ties":
        return rng.integers(0, 2, m).astype(np.float32)
    if kind == "equal":      # every pair ties at first
        return np.full(m, 7, np.float32)
    if kind == "scales":     # magnitudes over 2^40
        return np.ldexp(rng.standard_normal(m), rng.integers(-20, 20, m)).astype(np.float32)
    raise ValueError(kind)


@pytest.mark.parametrize("order", ["symmetric", "linear"])
@pytest.mark.parametrize("n,kind", [(2, "scores"), (63, "ties"), (64, "scores"), (65, "equal"), (128, "balanced"),
                                    (229, "scales"), (230, "ties"), (231, "scores"), (232, "equal"), (383, "ties"),
                                    (384, "balanced"), (640, "scales"), (1025, "scores"), (1400, "balanced")])
def test_join_kernels_match_oracle(gpu, n, kind, order):
    tri = _matrix(n, kind, np.random.default_rng(5000 + n))
    got = phylogeny.run_triangle(tri, n, order=_lib.MSA_NJ_LINEAR if order == "linear" else _lib.MSA_NJ_SYMMETRIC)
    _same(got, O.oracle_nj(tri, n, order))


def _spotted(n, value):
    rng = np.random.default_rng(n)
    tri = np.round(rng.normal(-50, 20, n * (n - 1) // 2)).astype(np.float32)
    tri[rng.integers(0, len(tri), 3)] = value
    return tri


@pytest.mark.parametrize("order", ["symmetric", "linear"])
@pytest.mark.parametrize("n", [40, 230, 300, 700])
@pytest.mark.parametrize("value", [1e20, 1e30, -3e37])
def test_huge_distances_match_oracle(gpu, n, value, order):
    """Values at which the bounds on Q lose their grip or are switched off."""
    tri = _spotted(n, value)
    got = phylogeny.run_triangle(tri, n, order=_lib.MSA_NJ_LINEAR if order == "linear" else _lib.MSA_NJ_SYMMETRIC)
    _same(got, O.oracle_nj(tri, n, order))


@pytest.mark.parametrize("order", [_lib.MSA_NJ_SYMMETRIC, _lib.MSA_NJ_LINEAR])
@pytest.mark.parametrize("n", [40, 200, 300, 700])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_non_finite_distances_match_the_full_scan(gpu, n, order, value):
    """The bounded search and the kernel that scans every pair take the same
    joins with the same length bits, or fail with the same status."""
    tri = _spotted(n, value)
    ctx = runtime.context(0)
    results = []
    for clusters in (0, 2):
        _lib.check(_lib.lib().msa_nj_set_clusters(ctx.handle, clusters, 8, 0, 0))
        try:
            t = phylogeny.run_triangle(tri, n, order=order)
            results.append([t.parent.tolist(), t.level.tolist(), t.distance.view(np.uint32).tolist()])
        except _lib.MsaError as e:
            results.append(e.status)
        finally:
            _lib.check(_lib.lib().msa_nj_set_clusters(ctx.handle, 0, 0, 0, 0))
    assert results[0] == results[1]
