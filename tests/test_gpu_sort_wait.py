"""Sorts whose look-back waits run out at once: the blocks count the earlier tiles themselves, and
every order is that of a sort that waited.  The point orders are compared with numpy's; the records
of the chain (event, rank, queue and node sorts) with those of a context that waits."""
import numpy as np
import pytest

import ehgp
import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wait", [0, 1, 5])
@pytest.mark.parametrize("n", [2049, 6145, 100003])
def test_point_orders(n, wait):
    rng = np.random.default_rng(n)
    pts = rng.random((n, 3))
    pts[::3, 0] = np.round(pts[::3, 0] * 8) / 8  # equal leading keys
    with ehgp.Context(max_points=n) as ctx:
        want = ctx.lbvh_build(pts)
        ctx.tune(ctx.TUNE_SORT_WAIT, wait)
        got = ctx.lbvh_build(pts)
    assert np.array_equal(got.source_index, np.lexsort((pts[:, 2], pts[:, 1], pts[:, 0])).astype(np.uint64))
    assert np.array_equal(got.leaves, want.leaves) and np.array_equal(got.nodes, want.nodes)


@pytest.mark.parametrize("pts", [workloads.uniform_cube(3001, 4),
                                 np.concatenate([workloads.uniform_cube(900, 2) + [i, 0, 0] for i in (0.0, 2.0, 4.0)])],
                         ids=["uniform", "copies"])
def test_chain_records(pts):
    pts = np.round(pts * 2.0**40) / 2.0**40  # the copies stay exact
    out = []
    for wait in (None, 0):
        with ehgp.Context(max_points=len(pts)) as ctx:
            if wait is not None:
                ctx.tune(ctx.TUNE_SORT_WAIT, wait)
            ctx.lbvh_build(pts, outputs=False)
            r = {**ctx.pairs(6), "higher": ctx.higher(6)}
            r.update(ctx.hierarchy(6))
            out.append({k: v for k, v in r.items() if isinstance(v, np.ndarray)})
    assert out[0].keys() == out[1].keys() and len(out[0]) > 8
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


def test_longer_waits_are_refused():
    with ehgp.Context(max_points=10) as ctx, pytest.raises(ehgp.InvalidArgument):
        ctx.tune(ctx.TUNE_SORT_WAIT, (1 << 20) + 1)
