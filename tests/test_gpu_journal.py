"""Forest journal on clouds made of exact translated copies of one tile: every event of a tile is
tied, level for level, with its copies, so that births and saddles share batches and the saddles
that join neighbouring copies share groups.  The records are whole numbers and equal the
restatement's; the first row of sizes has no tie at all, the last more copies than points."""
import numpy as np
import pytest

import ehgp
from geomcheck import gpu_hierarchy_text, hierarchy_diff
from oracle import pyoracle

CASES = [(1, 7, 10), (2, 3, 10), (2, 14, 4), (3, 9, 10), (4, 8, 3), (3, 12, 2), (9, 3, 10)]


def copies(count: int, tile: int) -> np.ndarray:
    """`count` copies of `tile` points on a 2^-20 grid, along an exact oblique step."""
    base = np.floor(np.random.default_rng(tile).random((tile, 3)) * 2.0**20) / 2.0**20
    return np.concatenate([base + i * np.array([1.125, 0.375, 0.21875]) for i in range(count)])


@pytest.mark.parametrize("count,tile,K", CASES)
def test_copies_tie_and_are_not_refused(count, tile, K):
    text = pyoracle.hierarchy(copies(count, tile), K)
    assert not text.rstrip().endswith("D 4 3 4")
    shared = [l for l in text.splitlines() if l[0] == "B"]
    assert shared  # batches are printed: the comparison below covers their records


@pytest.mark.gpu
@pytest.mark.parametrize("count,tile,K", CASES)
def test_gpu_journal_of_tied_copies(count, tile, K):
    pts = copies(count, tile)
    with ehgp.Context(max_points=64) as ctx:
        ctx.lbvh_build(pts, outputs=False)
        got, want = gpu_hierarchy_text(ctx, K), pyoracle.hierarchy(pts, K)
    assert got == want, hierarchy_diff(got, want)
