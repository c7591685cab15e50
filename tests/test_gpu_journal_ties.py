"""The tied copies of test_gpu_journal.py do tie: batches with several saddles, groups that join several
with three copies and more, neither without copies; and a cloud whose saddles in shared batches are more than one block
sorts (2,048), against the restatement."""
import numpy as np
import pytest

import ehgp
from geomcheck import gpu_hierarchy_text, hierarchy_diff
from oracle import pyoracle
from test_gpu_journal import CASES, copies


def shares(text: str) -> tuple[int, int, int]:
    """Most saddles of a batch and of a group, and the saddles in batches of several."""
    batches = [int(l.split()[-1]) for l in text.splitlines() if l[0] == "J"]
    groups = [int(l.split()[4]) for l in text.splitlines() if l[0] == "G"]
    return max(batches), max(groups), sum(b for b in batches if b > 1)


@pytest.mark.parametrize("count,tile,K", CASES)
def test_copies_share_batches_and_groups(count, tile, K):
    batch, group, shared = shares(pyoracle.hierarchy(copies(count, tile), K))
    if count == 1:
        assert (batch, group, shared) == (1, 1, 0)
    else:
        assert batch > 1 and shared > 0 and (group > 1 or count == 2)


@pytest.mark.gpu
def test_gpu_journal_of_many_shared_saddles():
    pts, K = copies(5, 20), 6
    want = pyoracle.hierarchy(pts, K)
    assert shares(want)[2] > 2048
    with ehgp.Context(max_points=len(pts)) as ctx:
        ctx.lbvh_build(pts, outputs=False)
        got = gpu_hierarchy_text(ctx, K)
    assert got == want, hierarchy_diff(got, want)
