"""Radix sorts at the edges of their tiles, through outputs whose order they decide: the canonical
point order and the Morton leaf order (the snapshot of the LBVH) against numpy and the oracle, for
sizes around one warp, the single-block limit, whole tiles and a remainder, with many equal keys."""
import numpy as np
import pytest

import ehgp
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def cloud(n: int, repeat: bool) -> np.ndarray:
    """n points in no order; with `repeat`, few values per coordinate (digits and keys repeat)."""
    rng = np.random.default_rng(n)
    if not repeat:
        return rng.standard_normal((n, 3))
    side = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side) - side // 2] * 3, indexing="ij"), -1).reshape(-1, 3)
    return rng.permutation(g[:n].astype(np.float64) / 4.0)


@pytest.mark.parametrize("repeat", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 2047, 2048, 2049, 4096, 6145, 20000])
def test_gpu_sorted_orders(n, repeat):
    pts = cloud(n, repeat)
    with ehgp.Context(max_points=n) as ctx:
        snap = ctx.lbvh_build(pts)
    order = np.lexsort((pts[:, 2], pts[:, 1], pts[:, 0]))
    assert np.array_equal(snap.source_index, order.astype(np.uint64))
    ref = pyoracle.lbvh_build(pts)
    assert np.array_equal(snap.leaves, ref["leaves"])
    codes = snap.leaves[:, 0]
    assert np.all((codes[:-1] < codes[1:]) | ((codes[:-1] == codes[1:]) & (snap.leaves[:-1, 1] < snap.leaves[1:, 1])))
