"""Clouds multiplied by powers of two: every predicate is homogeneous, so the records are the same.
Far below 1 the binary32 pruning tests see products that underflow.  Below the range of binary32
itself the index's boxes hold no shape any more, and a cloud may be refused for its traversals'
capacity, but its records are never others."""
import numpy as np
import pytest

import ehgp
import workloads

pytestmark = pytest.mark.gpu

CLOUDS = {"uniform300": workloads.uniform_cube(300, 3), "uniform1500": workloads.uniform_cube(1500, 8),
          "clustered600": workloads.clustered(600, 3)}


def scaled(pts, e):
    return np.ldexp(np.floor(pts * 2.0**30), e - 30)


@pytest.mark.parametrize("name", CLOUDS)
@pytest.mark.parametrize("K", [3, 10])
def test_pairs_do_not_depend_on_the_unit(name, K):
    pts = CLOUDS[name]
    out = {}
    with ehgp.Context(max_points=len(pts)) as ctx:
        for e in (0, -500, -140, -100, -80, -74, -72, -70, -68, -66, -64, -60, -40, -20, 20, 40, 60, 90):
            ctx.lbvh_build(scaled(pts, e), outputs=False)
            try:
                r = ctx.pairs(K)
            except ehgp.CapacityError:
                assert e < -149
                continue
            out[e] = r["records"].tobytes()
            if e <= 0:  # squared lengths in units of the cloud's own grid
                out[e] += r["level_num"].tobytes()
            assert out[e] == out[0][:len(out[e])], e


@pytest.mark.parametrize("name", ["uniform300", "clustered600"])
def test_hierarchies_do_not_depend_on_the_unit(name):
    pts = CLOUDS[name]
    with ehgp.Context(max_points=len(pts)) as ctx:
        want = None
        for e in (0, -100, -90, -80, -74, -70, -66, -62, -58, -40, 20, 60):
            ctx.lbvh_build(scaled(pts, e), outputs=False)
            got = ctx.hierarchy(6)
            want = want or got
            for k, v in want.items():
                assert not isinstance(v, np.ndarray) or np.array_equal(got[k], v), (e, k)
