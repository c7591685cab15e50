"""Device memory: what a context reports covers the hierarchy's arrays and records, and a server's
requests wait while theirs do not fit its share, whatever idle workers still hold."""
import threading
import time

import numpy as np
import pytest

import ehgp
import workloads

pytestmark = pytest.mark.gpu

SIDE = 20


def _used():
    import torch
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.fixture(scope="module", autouse=True)
def driver_memory():
    """One small chain first: the driver keeps local memory for the kernels' stacks (1.3 GB)."""
    with ehgp.Context(max_points=1000) as ctx:
        ctx.lbvh_build(workloads.jittered_lattice(10, 1), outputs=False)
        ctx.hierarchy(10)


def test_device_bytes_cover_the_hierarchy():
    pts = workloads.jittered_lattice(SIDE, 1)
    before = _used()
    with ehgp.Context(max_points=len(pts)) as ctx:
        base = ctx.device_bytes
        ctx.lbvh_build(pts, outputs=False)
        for K in (4, 10):
            r = ctx.hierarchy(K)
            records = sum(v.nbytes for k, v in r.items() if isinstance(v, np.ndarray))
            assert ctx.device_bytes - base > records
        used = _used() - before  # whole pages per buffer
        assert used - ctx.device_bytes < 0.05 * ctx.device_bytes + (256 << 20)
        assert ctx.counters()["device_bytes"] == ctx.device_bytes
    assert _used() - before < 256 << 20


def test_server_requests_wait_for_the_whole_footprint():
    pts = workloads.jittered_lattice(SIDE, 1)
    n, workers = len(pts), 6
    with ehgp.Context(max_points=n) as ctx:
        ctx.lbvh_build(pts, outputs=False)
        base = ctx.device_bytes
        ctx.pairs(10), ctx.higher(10)
        records = ctx.device_bytes - base  # record buffers that grew stay with their worker
        ctx.hierarchy(10)
        whole = ctx.device_bytes
    import torch
    total = torch.cuda.get_device_properties(0).total_memory
    budget = 2.8 * whole  # two requests and not three
    most, stop = [0], threading.Event()
    with ehgp.Server(workers=workers, max_points=n, hbm_fraction=budget / total) as srv:
        start = _used()

        def watch():
            while not stop.is_set():
                most[0] = max(most[0], _used() - start)
                time.sleep(0.002)

        t = threading.Thread(target=watch)
        t.start()
        try:
            ids = [srv.submit(pts, 10) for _ in range(10)]
            first = None
            for rid in ids:
                assert srv.wait(rid) == 0, srv.info(rid)["error"]
                if rid in (ids[0], ids[-1]):
                    got = srv.result(rid)
                    first = first or got
                    assert all(np.array_equal(got[k], first[k]) for k in first)
                srv.release(rid)
        finally:
            stop.set()
            t.join()
        assert srv.stats()["memory_waits"] > 0
    assert most[0] < budget + workers * (records + (128 << 20))


def _arrays(ctx, K):
    r = {k: v for k, v in ctx.hierarchy(K).items() if isinstance(v, np.ndarray)}
    r["supports"] = ctx.event_supports(r["nodes"]["level_event"])
    return r


@pytest.mark.parametrize("pts", [workloads.jittered_lattice(10, 2),
                                 np.concatenate([np.round(workloads.uniform_cube(150, 5) * 2.0**30) / 2.0**30 + [i, 0, 0]
                                                 for i in (0.0, 2.0, 4.0)])], ids=["lattice", "copies"])
def test_hierarchies_without_room_on_the_device(pts):
    """Blocks above 8 MB (more than any one array needs, less than the journal) are refused: the descent
    runs in parts, the records go to host memory."""
    with ehgp.Context(max_points=len(pts)) as ctx:
        ctx.lbvh_build(pts, outputs=False)
        want = _arrays(ctx, 10)
        roomy = ctx.device_bytes
        for block in (8 << 20, 8 << 20, 0, 8 << 20):
            ctx.tune(ctx.TUNE_HIERARCHY_BLOCK, block)
            got = _arrays(ctx, 10)
            assert got.keys() == want.keys()
            for k in want:
                assert np.array_equal(got[k], want[k]), (block, k)
            assert (ctx.device_bytes < 0.8 * roomy) == (block > 0)
        ctx.tune(ctx.TUNE_HIERARCHY_BLOCK, 4096)  # no room for anything
        with pytest.raises(ehgp.EhgpError) as e:
            ctx.hierarchy(10)
        assert e.value.status == 4
        ctx.tune(ctx.TUNE_HIERARCHY_BLOCK, 0)
        got = _arrays(ctx, 10)
        assert all(np.array_equal(got[k], want[k]) for k in want)
