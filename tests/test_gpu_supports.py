"""Edges of the support and descent launches against the oracle: clouds around the length of a
warp's witness list, walks long enough to be handed over, tied clouds that binary64 leaves open,
and facets whose miniball holds more points than the facet.  Every record is whole numbers or an
exact level, so each comparison is equality."""
import numpy as np
import pytest

import workloads
from geomcheck import gpu_hierarchy_text, gpu_higher_records, gpu_pair_records, hierarchy_diff, higher_match, pairs_match
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def shell(n: int) -> np.ndarray:
    """n points within 1e-3 of a sphere: far pairs see nearly the whole cloud from their ball."""
    rng = np.random.default_rng(n)
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True) * (1.0 + 1e-3 * rng.random((n, 1)))


def grid(n: int, steps: int) -> np.ndarray:
    """About n points, every second one on a coarse grid: equal levels and cospherical points."""
    p = np.random.default_rng(n).random((n, 3))
    p[::2] = np.round(p[::2] * steps) / steps
    return np.unique(p, axis=0)


def nested(n: int) -> np.ndarray:
    """Two tight clusters and points between them: balls of wide facets hold more than k points."""
    rng = np.random.default_rng(n)
    a = 1e-3 * rng.random((n // 3, 3))
    b = 1e-3 * rng.random((n // 3, 3)) + [1.0, 0.5, 0.25]
    return np.concatenate([a, b, rng.random((n - 2 * (n // 3), 3))])


def canonical(ctx, pts):
    snap = ctx.lbvh_build(pts)
    return np.asarray(pts, np.float64)[snap.source_index.astype(np.int64)]


@pytest.mark.parametrize("n", [12, 31, 32, 33, 63, 64, 65, 66, 97])
@pytest.mark.parametrize("K", [1, 10])
def test_pairs_around_the_witness_list(ctx, n, K):
    P = canonical(ctx, workloads.uniform_cube(n, n))
    pairs_match(gpu_pair_records(ctx, K, P), pyoracle.pairs(P, K))


@pytest.mark.parametrize("pts", [shell(1200), grid(400, 6)], ids=["shell1200", "grid400"])
def test_pairs_of_long_walks(ctx, pts):
    P = canonical(ctx, pts)
    pairs_match(gpu_pair_records(ctx, 10, P), pyoracle.pairs(P, 10))


@pytest.mark.parametrize("pts,K", [(grid(48, 2), 10), (grid(64, 3), 4), (shell(56), 10), (nested(60), 10), (nested(33), 2)],
                         ids=["grid48", "grid64_K4", "shell56", "nested60", "nested33_K2"])
def test_higher_supports_left_open_in_binary32(ctx, pts, K):
    P = canonical(ctx, pts)
    higher_match(gpu_higher_records(ctx, K, P), pyoracle.higher(P, K))


@pytest.mark.parametrize("n,K", [(24, 10), (36, 4), (45, 2), (30, 3)])
def test_descents_with_more_inside_points_than_the_facet(ctx, n, K):
    pts = nested(n)
    ctx.lbvh_build(pts, outputs=False)
    got, want = gpu_hierarchy_text(ctx, K), pyoracle.hierarchy(pts, K)
    assert got == want, hierarchy_diff(got, want)
