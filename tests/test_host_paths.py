"""CPU: the host paths of libgravcuda.so on a runtime that needs no GPU
(fake_cudart.cpp, preloaded in a child process): what they do with device
memory when an allocation fails, and how they launch."""
import json
import os
import subprocess
import sys

import pytest

from conftest import PKG_ROOT, REPO

# a two-body plan built on the (fake) device, evaluated, and its adjoint; returns the status
PRELUDE = """
import ctypes, json, os, sys
sys.path.insert(0, {pkg!r})
import numpy as np
from pgrav import gravcuda as gc
from pgrav.host import Params
L = gc.lib()
fake = ctypes.CDLL({fake!r})
fake.fake_allocs_before.restype = ctypes.c_long
bodies = np.zeros((16, 4), np.float32)
at = bodies.ctypes.data + -bodies.ctypes.data % 16
def counts():
    c = (ctypes.c_long * 6)()
    fake.fake_counts(c)
    return dict(zip(("allocs", "live", "double", "trims", "pending", "error"), c))
def used():
    b = (ctypes.c_long * 2)()
    fake.fake_bytes(b)
    return list(b)
def build(box, tuning=None, n=2):
    data = at
    if n > 2:
        many = np.zeros((n + 1, 4), np.float32)
        data = many.ctypes.data + -many.ctypes.data % 16
    t = ctypes.byref(gc.Tuning(*tuning)) if tuning else None
    p = Params(16, 32, 7, 20, 1e-3, 0.0, 0.0, box, 0, 0, 0.2, 0.0)
    h = ctypes.c_void_p()
    rc = L.grav_plan_build_CUDA(ctypes.byref(p), data, n, 1e-4, 1.0, int(box > 0), t, ctypes.byref(h))
    if rc == 0 and n == 2:
        rc = L.grav_groups_eval_CUDA(h, None) or L.grav_plan_adjoint_CUDA(h, at, at, None)
    return rc, h
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from pgrav import _build
    _build.build_all()
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run([_build._cxx(), "-O1", "-std=c++17", "-fPIC", "-shared", "-o", so,
                    os.path.join(REPO, "tests", "fake_cudart.cpp")], check=True)

    def go(body):
        code = PRELUDE.format(pkg=PKG_ROOT, fake=so) + body
        r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600,
                           env=dict(os.environ, LD_PRELOAD=so))
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout.splitlines()[-1])

    return go


# every allocation of a call fails in turn: status and memory counts of each
FAIL_EACH = """
res = []
for box in (0.0, 1.0):
    fake.fake_reset(0, 0)
    rc, h = build(box)
    assert rc == 0, rc
    last, queue = counts()["allocs"], fake.fake_allocs_before(b"k_queue_count")
    L.grav_plan_free(h)
    assert counts()["live"] == 0
    for k in {range}:
        fake.fake_reset(k, 0)
        rc, h = build(box)
        if h:
            L.grav_plan_free(h)
        L.gravcuda_clear_status()
        fake.cudaGetLastError()
        res.append([box, k, rc, counts()])
print(json.dumps(res))
"""


def check_freed_once(out):
    assert len(out) >= 40
    for box, k, rc, c in out:
        assert rc != 0 and c["double"] == 0 and c["live"] == 0, (box, k, rc, c)


def test_a_failed_plan_frees_every_buffer_once(run):
    """The work queue of a device-built tree, the plan around it, its
    evaluation and adjoint: the k-th allocation fails, for every k."""
    check_freed_once(run(FAIL_EACH.format(range="range(queue + 1, last + 1)")))


def test_a_failed_tree_frees_every_buffer_once(run):
    """The tree, its tables and its lists: the k-th allocation fails."""
    check_freed_once(run(FAIL_EACH.format(range="range(1, queue + 1)")))


def test_a_failed_call_does_not_fail_the_next(run):
    """A build after one whose k-th allocation failed succeeds, for every k."""
    out = run("""
res = []
fake.fake_reset(0, 0)
rc, h = build(0.0)
total = counts()["allocs"]
L.grav_plan_free(h)
for k in range(1, total + 1):
    fake.fake_reset(k, 0)
    rc, h = build(0.0)
    if h:
        L.grav_plan_free(h)
    L.gravcuda_clear_status()
    fake.fake_reset(0, 0)
    again, h = build(0.0)
    if h:
        L.grav_plan_free(h)
    L.gravcuda_clear_status()
    fake.cudaGetLastError()
    res.append([k, rc, again])
print(json.dumps(res))
""")
    assert len(out) >= 60
    for k, failed, again in out:
        assert failed != 0 and again == 0, (k, failed, again)


def test_the_pool_gives_its_reserve_back_first(run):
    """The k-th allocation of a build, an evaluation and an adjoint fails until
    the pool has given back what it keeps reserved: every call succeeds."""
    out = run("""
res = []
for box in (0.0, 1.0):
    fake.fake_reset(0, 0)
    rc, h = build(box)
    total = counts()["allocs"]
    L.grav_plan_free(h)
    for k in range(1, total + 1):
        fake.fake_reset(k, 1)
        rc, h = build(box)
        res.append([box, k, rc, counts()])
        if h:
            L.grav_plan_free(h)
        L.gravcuda_clear_status()
print(json.dumps(res))
""")
    assert len(out) >= 150
    for box, k, rc, c in out:
        assert rc == 0 and c["trims"] == 1, (box, k, rc, c)


def test_a_block_cap_counts_blocks_of_the_given_warps(run):
    """blocks_per_sm caps the list kernels' resident warps at that many blocks
    of warps_per_block warps, whatever blocks they run in (three blocks fit an
    SM of 148 here)."""
    caps = {"8,0": 3, "8,1": 2, "8,2": 3, "4,1": 1, "4,2": 2, "4,4": 3, "2,1": 1, "2,2": 2, "5,1": 2}
    out = run("""
res = []
for w, b in %r:
    rc, h = build(0.0, (w, 0, 0, 0, b, 0, 0))
    assert rc == 0
    res.append([w, b, [fake.fake_grid(k) for k in (b"k_points", b"k_cells")]])
    L.grav_plan_free(h)
print(json.dumps(res))
""" % ([[int(x) for x in k.split(",")] for k in caps],))
    for w, b, grids in out:
        assert grids == [caps[f"{w},{b}"] * 148] * 2, (w, b, grids)


def test_cell_arrays_hold_what_the_leaves_can_make(run):
    """A plan of n bodies in leaves of L holds its bodies (16 bytes each), their
    order (8), its results (16), the links of at most 7 n / L cells (20) and
    little more, and a tree that would need more cells than list indices can
    name is refused as such, after a bounded search for room."""
    n = 3_000_000
    held, refused, message = run("""
n = %d
rc, h = build(0.0, n=n)
assert rc == 0
held = used()[0]
L.grav_plan_free(h)
fake.fake_reset(0, 0)
fake.fake_cells(ctypes.c_longlong(1 << 40))
rc, h = build(0.0, n=n)
print(json.dumps([held, rc, L.gravcuda_status_string().decode()]))
""" % n)
    assert held < (40 + 20 * 7 / 16) * n + (4 << 20), held
    assert refused == -1 and "27-bit" in message, (refused, message)


def test_sink_buffers_are_given_back_between_walks(run):
    """The drop-in keeps its sink buffers for the next walk;
    grav_groups_release_CUDA returns them, but not under a registered table."""
    n = 100_000
    idle, kept, released, again, registered, final = run("""
n = %d
btab = np.zeros((n, 16), np.float32)
res = []
L.CUDA_Init(None)
res.append(used()[0])
L.WalkInitSinkCUDA(btab.ctypes.data, 16, n)
L.WalkTerminateSinkCUDA(btab.ctypes.data, 16, n)
res.append(used()[0])
L.grav_groups_release_CUDA()
res.append(used()[0])
L.WalkInitSinkCUDA(btab.ctypes.data, 16, n)
res.append(used()[0])
L.grav_groups_release_CUDA()
res.append(used()[0])
L.WalkTerminateSinkCUDA(btab.ctypes.data, 16, n)
L.CUDA_Finalize()
res.append(used()[0])
assert L.gravcuda_status() == 0 and counts()["double"] == 0
print(json.dumps(res))
""" % n)
    assert kept == again == registered == idle + 28 * n
    assert released == idle and final == 0


def test_a_new_plan_leaves_nothing_on_the_default_stream(run):
    """Streams other than the default one do not wait for it, so a plan's
    tables and cleared words are complete when the call that makes them
    returns: uploaded with copied lists and with lists in host memory, built
    on the device, retuned, and with its tree links set."""
    out = run("""
from pgrav import ics, host
res = {}
pos, m = ics.grf_box(12, seed=1)
t = host.Tree(pos, m, box=1.0, leaf_max=16, group_max=32, p2cut=7, p4cut=8, tol=1e-4)
for in_host in (0, 1):
    p = gc.Problem()
    p.nbodies, p.ncells, p.ngroups = t.n, t.ncells, t.ngroups
    p.points, p.qcells, p.hcells, p.groups = (a.ctypes.data for a in (t.points, t.qcells, t.hcells, t.groups))
    p.pptr, p.qptr, p.hptr, p.cptr = (a.ctypes.data for a in t.ptr)
    p.plist, p.qlist, p.hlist, p.clist = (a.ctypes.data for a in (t.plist, t.qlist, t.hlist, t.clist))
    p.eps2, p.box, p.ewald, p.quad_phi_sign, p.lists_in_host = 1e-4, 1.0, 1, 1.0, in_host
    h = ctypes.c_void_p()
    fake.fake_reset(0, 0)
    rc = L.grav_groups_upload_CUDA(ctypes.byref(p), None, ctypes.byref(h))
    res["upload %d" % in_host] = [rc, counts()["pending"]]
    rc = L.grav_plan_retune_CUDA(h, ctypes.byref(gc.Tuning(4, 256, 128, 64, 0, 0, 0)))
    res["retune %d" % in_host] = [rc, counts()["pending"]]
    links = t.cell_ranges() + t.cell_links()
    rc = L.grav_plan_set_tree_CUDA(h, *(x.ctypes.data for x in links))
    res["set_tree %d" % in_host] = [rc, counts()["pending"]]
    L.grav_plan_free(h)
fake.fake_reset(0, 0)
p = Params(16, 32, 7, 20, 1e-3, 0.0, 0.0, 1.0, 0, 0, 0.2, 0.0)
h = ctypes.c_void_p()
rc = L.grav_plan_build_CUDA(ctypes.byref(p), at, 2, 1e-4, 1.0, 1, None, ctypes.byref(h))
res["build"] = [rc, counts()["pending"]]
rc = L.grav_plan_retune_CUDA(h, ctypes.byref(gc.Tuning(4, 256, 128, 64, 0, 0, 0)))
res["retune built"] = [rc, counts()["pending"]]
L.grav_plan_free(h)
print(json.dumps(res))
""")
    for call, (rc, pending) in out.items():
        assert rc == 0 and pending == 0, (call, rc, pending)


def test_a_plan_of_small_blocks_leaves_the_others_their_shared_memory(run):
    """A kernel's shared memory limit is the process's: a plan of one-warp
    blocks, evaluated between another thread's setting it and its launch,
    must not lower it."""
    out = run("""
res = []
for w in (8, 1, 4):
    rc, h = build(0.0, (w, 0, 0, 0, 0, 0, 0))
    assert rc == 0
    res.append([fake.fake_smem_limit(k) for k in (b"k_pointsILb0", b"k_cellsILi1ELb0")])
    L.grav_plan_free(h)
print(json.dumps(res))
""")
    assert min(out[0]) > 0 and out[0] == out[1] == out[2]


def test_a_plan_without_its_queue_is_not_evaluated(run):
    """A retune whose k-th allocation fails leaves a plan that refuses to be
    evaluated or differentiated (its kernels would read null queues), and that
    another retune makes whole."""
    out = run("""
t = ctypes.byref(gc.Tuning(4, 256, 128, 64, 0, 0, 0))
rc, h = build(0.0)
fake.fake_reset(0, 0)
assert rc == 0 and L.grav_plan_retune_CUDA(h, t) == 0
total, res = counts()["allocs"], []
for k in range(1, total + 1):
    fake.fake_reset(k, 0)
    failed = L.grav_plan_retune_CUDA(h, t)
    fake.fake_reset(0, 0)
    res.append([k, failed, L.grav_groups_eval_CUDA(h, None), L.grav_plan_adjoint_CUDA(h, at, at, None),
                fake.fake_allocs_before(b"k_points"), L.grav_plan_retune_CUDA(h, t),
                L.grav_groups_eval_CUDA(h, None)])
L.grav_plan_free(h)
print(json.dumps(res))
""")
    assert len(out) >= 5
    for k, failed, ev, adj, launched, again, after in out:
        assert failed and ev == -1 and adj == -1 and launched == -1, (k, failed, ev, adj, launched)
        assert again == 0 and after == 0


def test_a_plan_is_freed_after_the_work_that_uses_it(run):
    """A device-built plan's buffers go back to the pool only when what was
    queued on another stream (an evaluation, an adjoint, a refit, a step) is
    done with them; a plan used on the default stream alone, in whose order they
    go back, does not hold the device up (a capture elsewhere would not survive
    that)."""
    out = run("""
res = []
fake.fake_freed_early.restype = fake.fake_device_waits.restype = ctypes.c_long
uses = {
    "eval": lambda h, st: L.grav_groups_eval_CUDA(h, st),
    "adjoint": lambda h, st: L.grav_plan_adjoint_CUDA(h, at, at, st),
    "refit": lambda h, st: L.grav_plan_refit_CUDA(h, st),
    "step": lambda h, st: L.grav_plan_step_CUDA(h, at, at, at, st, 0),
}
for box in (0.0, 1.0):
    for name, use in uses.items():
        for stream in (0x5000, None):
            rc, h = build(box)
            fake.cudaDeviceSynchronize()
            fake.fake_reset(0, 0)
            assert rc == 0 and use(h, stream) == 0
            L.grav_plan_free(h)
            res.append([name, stream is None, fake.fake_freed_early(), fake.fake_device_waits(),
                        counts()["live"]])
print(json.dumps(res))
""")
    assert len(out) == 16
    for name, default, early, waits, live in out:
        assert early == 0 and live == 0 and waits == (0 if default else 1), (name, default, early, waits)
