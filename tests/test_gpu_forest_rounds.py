"""Forest journal where its rounds are many: on points whose spacing shrinks along a curve, every
component's nearest partner is younger, so one component dies per round.  What the rounds leave is
applied in order on the host; the records do not depend on how many rounds the device is given."""
import numpy as np
import pytest

import ehgp
import workloads
from geomcheck import gpu_hierarchy_text, hierarchy_diff
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def shrinking(n, turn=0.0):
    """n points whose spacing shrinks, on a line or (turn > 0) a helix, oldest first."""
    t = np.sqrt(np.arange(1.0, n + 1.0))
    return np.c_[t, np.cos(turn * t) * turn, np.sin(turn * t) * turn]


def copies(count, tile):
    base = np.floor(np.random.default_rng(tile).random((tile, 3)) * 2.0**20) / 2.0**20
    return np.concatenate([base + i * np.array([1.125, 0.375, 0.21875]) for i in range(count)])


CLOUDS = {"uniform": (workloads.uniform_cube(1201, 3), 10), "lattice": (workloads.jittered_lattice(16, 2), 6),
          "mixture": (workloads.mixture_cloud(1501, np.random.Generator(np.random.PCG64(4))), 10),
          "copies": (copies(30, 17), 10), "line": (shrinking(9001), 4), "helix": (shrinking(1801, 0.5), 10)}


@pytest.mark.parametrize("name", CLOUDS)
def test_records_do_not_depend_on_the_rounds(name):
    pts, K = CLOUDS[name]
    with ehgp.Context(max_points=len(pts)) as ctx:
        ctx.lbvh_build(pts, outputs=False)
        want = ctx.hierarchy(K)
        assert (ctx.counters()["forest_rest"] > 0) == (name in ("line", "helix"))
        for rounds in (0, 1, 4, 13):
            ctx.tune(ctx.TUNE_FOREST_ROUNDS, rounds)
            got = ctx.hierarchy(K)
            assert rounds > 0 or ctx.counters()["forest_rest"] > 0
            for k, v in want.items():
                assert not isinstance(v, np.ndarray) or np.array_equal(got[k], v), (rounds, k)


@pytest.mark.parametrize("pts,K", [(workloads.uniform_cube(33, 5), 10), (copies(3, 9), 10), (shrinking(40), 3)],
                         ids=["uniform33", "copies27", "line40"])
def test_families_applied_on_the_host(pts, K):
    with ehgp.Context(max_points=64) as ctx:
        ctx.tune(ctx.TUNE_FOREST_ROUNDS, 0)
        ctx.lbvh_build(pts, outputs=False)
        got, want = gpu_hierarchy_text(ctx, K), pyoracle.hierarchy(pts, K)
        assert ctx.counters()["forest_rest"] > 0
    assert got == want, hierarchy_diff(got, want)


def test_a_chain_of_ever_older_partners_takes_no_round_each():
    """20,000 points on a line: 0.57 s with a device round per point."""
    pts = shrinking(20000)
    with ehgp.Context(max_points=len(pts)) as ctx:
        ctx.lbvh_build(pts, outputs=False)
        for _ in range(2):
            r = ctx.hierarchy(1)
        assert ctx.hier_stats()["forest_ms"] < 60.0
        assert len(r["nodes"]) == 2 * len(pts) - 1 and (r["nodes"]["kind"] == 2).sum() == len(pts) - 1
