"""Hand-over of long pair walks when the list of handed-over walks runs full: the records are those
of a context with ample room, whatever the list holds.  Clusters with a sparse background have
walks that are handed over by the thousand; the counters say that they were, and that the list was
full where it is meant to be."""
import numpy as np
import pytest

import ehgp
import workloads

pytestmark = pytest.mark.gpu

CLOUDS = {
    "clustered2003": lambda: workloads.clustered(2003, 5),
    "clustered8009": lambda: workloads.clustered(8009, 1),
    "mixture5003": lambda: workloads.mixture_cloud(5003, np.random.Generator(np.random.PCG64(2))),
    "clustered12007": lambda: workloads.clustered(12007, 3),
}


def _run(ctx, K):
    r = ctx.pairs(K)
    _, stats = ctx.kernel_stats()
    return r["records"].tobytes(), r["level_num"].tobytes(), int(stats[5]), int(stats[6])


@pytest.mark.parametrize("name", CLOUDS)
def test_records_do_not_depend_on_the_room_for_handed_over_walks(name):
    pts = CLOUDS[name]()
    n = len(pts)
    with ehgp.Context(max_points=8 * n) as ctx:
        ctx.lbvh_build(pts, outputs=False)
        want = _run(ctx, 10)
        assert want[2] == 0 and want[3] > 1000  # ample room, and walks that use it
        full = 0
        for room in (0, 1, 7, 255, 1000, 2 * n + 4096):
            ctx.tune(ctx.TUNE_PAIR_TASKS, room)
            ctx.lbvh_build(pts, outputs=False)  # the records are resident for one cloud and K
            got = _run(ctx, 10)
            assert got[:2] == want[:2], room
            assert room > 1000 or got[2] > 0, room
            full += got[2] > 0
        assert full >= 5


def test_room_above_the_list_is_refused():
    with ehgp.Context(max_points=100) as ctx:
        ctx.tune(ctx.TUNE_PAIR_TASKS, 2 * 100 + 4096)
        with pytest.raises(ehgp.InvalidArgument):
            ctx.tune(ctx.TUNE_PAIR_TASKS, 2 * 100 + 4097)


def test_points_on_a_line():
    """Walks that look at few boxes: 2.1 ms for these when each of them cost a step per witness."""
    n = 50000
    pts = np.zeros((n, 3))
    pts[:, 0] = np.sqrt(np.arange(1.0, n + 1.0))
    with ehgp.Context(max_points=n) as ctx:
        ctx.lbvh_build(pts, outputs=False)
        for _ in range(3):
            r = ctx.pairs(2)["records"]
        assert ctx.kernel_stats()[0] < 1.0
    u, v = r["u"].astype(np.int64), r["v"].astype(np.int64)
    want = sorted([(i, i + 1) for i in range(n - 1)] + [(i, i + 2) for i in range(n - 2)])
    assert np.array_equal(np.c_[u, v], np.array(want)) and np.array_equal(r["interior_count"], v - u - 1)
    assert np.array_equal(r["interior_ids"][v - u == 2, 0], u[v - u == 2] + 1)
