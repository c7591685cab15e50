"""Failures on the host's side of the library, made by a preloaded shim (host_faults.cpp): no
device call is made before the context's device is selected, a poisoned context hands nothing out,
and an allocation that fails is a status at the C interface, never an exception through it."""
import os
import subprocess
import sys

import pytest

import ehgp

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
PRELUDE = """
import ctypes as C, sys
sys.path[:0] = [%r, %r]
import numpy as np, ehgp, workloads
shim = C.CDLL(%r)
pts = workloads.jittered_lattice(16, 1)
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    ehgp.load()
    runtime = next(l.split()[-1] for l in open("/proc/self/maps") if "libcudart.so" in l)
    path = str(tmp_path_factory.mktemp("shim") / "host_faults.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", os.path.join(HERE, "host_faults.cpp"), "-o", path,
                    "-Wl,--no-as-needed", runtime, f"-Wl,-rpath,{os.path.dirname(runtime)}", "-ldl"], check=True)
    return path


def run(shim, code):
    body = PRELUDE % (os.path.dirname(HERE), os.path.join(os.path.dirname(HERE), "e-hgp_b200"), shim) + code
    r = subprocess.run([sys.executable, "-c", body], env={**os.environ, "LD_PRELOAD": shim}, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_copies_select_their_device_first(shim):
    run(shim, """
import threading
with ehgp.Context(max_points=len(pts)) as ctx:
    ctx.lbvh_build(pts, outputs=False)
    want = ctx.hierarchy(10)
    bufs = {f: np.zeros(max(ctx.last_hier_counts[c], 1), dt) for f, dt, c in ehgp._HIER_FIELDS}
    ho = ehgp.HierOut(*[b.ctypes.data for b in bufs.values()])
    assert sum(b.nbytes for b in bufs.values()) > 64 << 20  # through the pinned ring
    levels = np.ascontiguousarray(want["nodes"]["level_event"])
    sup = np.zeros((len(levels), 5), np.uint32)
    seen = []
    def copy():  # a thread of its own: no device selected yet
        shim.hf_watch(1)
        ctx._check(ctx.lib.ehgp_hier_copy(ctx._h, C.byref(ho)))
        seen.append(shim.hf_early_calls())
        shim.hf_watch(1)
        ctx._check(ctx.lib.ehgp_event_supports(ctx._h, levels.ctypes.data, len(levels), sup.ctypes.data))
        seen.append(shim.hf_early_calls())
        shim.hf_watch(0)
    t = threading.Thread(target=copy)
    t.start(); t.join()
    assert seen == [0, 0], seen
    for f, b in bufs.items():
        assert np.array_equal(b[:len(want[f])], want[f]), f
""")


def test_a_poisoned_context_hands_nothing_out(shim):
    run(shim, """
with ehgp.Context(max_points=len(pts)) as ctx:
    ctx.lbvh_build(pts, outputs=False)
    ctx.hierarchy(4)
    shim.hf_fail_sync()
    try:
        ctx.lbvh_build(pts, outputs=False)
        raise SystemExit("the failure was not reported")
    except ehgp.EhgpError as e:
        assert e.status == 8, e
    bufs = {f: np.zeros(max(ctx.last_hier_counts[c], 1), dt) for f, dt, c in ehgp._HIER_FIELDS}
    ho = ehgp.HierOut(*[b.ctypes.data for b in bufs.values()])
    assert ctx.lib.ehgp_hier_copy(ctx._h, C.byref(ho)) == 9
    lev = np.zeros(1, np.uint32); sup = np.zeros(5, np.uint32)
    assert ctx.lib.ehgp_event_supports(ctx._h, lev.ctypes.data, 1, sup.ctypes.data) == 9
    assert not any(b.view(np.uint8).any() for b in bufs.values())
""")


def test_failed_allocations_are_a_status(shim):
    """Every allocation of every call fails once; the call then says so, or did without; the next one works."""
    run(shim, """
def every(call, limit=300):
    said = 0
    for after in range(limit):
        shim.hf_fail_new(C.c_long(after))
        st = call()
        if not shim.hf_new_failed():
            assert st == 0, st
            return said
        assert st in (0, 4), st
        said += st == 4
    raise SystemExit("more allocations than looked at")
pts = workloads.jittered_lattice(12, 1)
with ehgp.Context(max_points=len(pts)) as ctx:
    lib, h = ctx.lib, ctx._h
    snap = ehgp.LbvhOut()
    nodes = np.zeros((2 * len(pts) - 1) * 80, np.uint8)
    snap.nodes = nodes.ctypes.data
    p64 = np.ascontiguousarray(pts, np.float64)
    every(lambda: lib.ehgp_lbvh_build(h, p64.ctypes.data, len(p64), C.byref(snap)))
    cnt = np.zeros(1, np.uint64)
    rec, lev = np.zeros(200000, ehgp.PAIR_RECORD), np.zeros((200000, 4), np.uint64)
    po = ehgp.PairsOut(rec.ctypes.data, lev.ctypes.data, len(rec), cnt.ctypes.data)
    every(lambda: lib.ehgp_pairs(h, 10, C.byref(po)))
    hrec = np.zeros(2000000, ehgp.HIGHER_RECORD)
    ho = ehgp.HigherOut(hrec.ctypes.data, len(hrec), cnt.ctypes.data)
    every(lambda: lib.ehgp_higher(h, 10, C.byref(ho)))
    hc = ehgp.HierCounts()
    every(lambda: lib.ehgp_hierarchy(h, 10, C.byref(hc)))
    want = ctx.hierarchy(10)
    bufs = {f: np.zeros(max(ctx.last_hier_counts[c], 1), dt) for f, dt, c in ehgp._HIER_FIELDS}
    out = ehgp.HierOut(*[b.ctypes.data for b in bufs.values()])
    every(lambda: lib.ehgp_hier_copy(h, C.byref(out)))
    for f, b in bufs.items():
        assert np.array_equal(b[:len(want[f])], want[f]), f
    events = np.ascontiguousarray(want["nodes"]["level_event"])
    sup = np.zeros((len(events), 5), np.uint32)
    every(lambda: lib.ehgp_event_supports(h, events.ctypes.data, len(events), sup.ctypes.data))
with ehgp.Server(workers=1, max_points=len(pts)) as srv:
    rid = srv.submit(pts, 10)
    assert srv.wait(rid) == 0
    want = srv.result(rid)
    got = {k: np.zeros_like(v) for k, v in want.items() if isinstance(v, np.ndarray)}
    out = ehgp.ServedOut(*[got[k].ctypes.data for k, _ in ehgp.ServedOut._fields_])
    every(lambda: srv.lib.ehgp_result_copy(srv._h, rid, C.byref(out)))
    for k in got:
        assert np.array_equal(got[k], want[k]), k
""")
