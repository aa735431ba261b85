"""The engine's host side when something runs out or overlaps, on a CUDA runtime
of host memory (tests/cpp/fake_cudart.cpp, loaded in front of the real one):
device and host allocations that fail, memory kept between calls, and calls on
several threads.  Kernels do not run here; what is checked is which calls
succeed, what stays allocated and that nothing ends the process.  Each case is a
process of its own."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

HEAD = """
import ctypes as C, sys, threading
sys.path[:0] = [{root!r} + "/gpu-smina_b200", {root!r} + "/tests"]
fake = C.CDLL({lib!r})
fake.fake_live.restype = C.c_size_t
fake.fake_limit.argtypes = [C.c_size_t]
import numpy as np
import smina_b200 as sb, workloads as W
T, R, gd, m = W.tables(), W.receptor(), W.box(), W.ligand()
HEAVY = [t for t in range(2, 27)]
def engine(precision=sb.PREC_FP32, tables=T, receptor=True):
    e = sb.Engine(0, precision)
    e.set_tables(tables)
    if receptor: e.set_receptor(0, R, gd)
    return e
def status(f, *a, **k):
    try:
        f(*a, **k)
        return sb.SG_OK
    except sb.SminaError as x:
        return x.code
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                        os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), "-pthread", "-o", lib],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def go(body):
        r = subprocess.run([sys.executable, "-c", HEAD.format(root=ROOT, lib=lib) + body], capture_output=True, text=True,
                           timeout=300, env=dict(os.environ, LD_PRELOAD=lib))
        assert r.returncode == 0, r.stdout + r.stderr
    return go


def test_dropped_maps_are_bounded(run):
    """Void maps wait for the next build in their place: freed by a direct sum
    there, by a drop and with the engine, and never more than 2 GiB."""
    run("""
e = engine()
x = W.random_confs(m, gd, 1, 1)
bare = fake.fake_live()
near = lambda: abs(fake.fake_live() - bare) < 2 << 20
def built():
    e.build_grids(0, HEAVY)
    assert fake.fake_live() > bare + (50 << 20)
grid = W.box(6.0)
void = (lambda: e.set_receptor(0, R, gd), lambda: e.set_tables(T),
        lambda: e.set_user_grid(0, grid, np.zeros(sb.grid_points(grid))))
direct = (lambda: e.minimize(0, [m], [0], x), lambda: e.refine(0, [m], [0], x), lambda: e.score(0, [m], [0], x),
          lambda: e.eval_direct(0, m, x))
for change in void:
    for use in direct:
        built(); change(); use(); assert near()
    built(); size = fake.fake_live(); change(); built(); assert abs(fake.fake_live() - size) < 2 << 20
sb.load().sg_drop_receptor(e._h, 0)
assert fake.fake_live() < bare
fake.fake_limit(64 << 30)
for k in range(16): e.set_receptor(k, R, W.box(36.0))
bare = fake.fake_live()
for k in range(16): e.build_grids(k, HEAVY)
assert fake.fake_live() > bare + (8 << 30)
e.set_tables(T)
assert bare < fake.fake_live() <= bare + (2 << 30)
e.close()
assert fake.fake_live() == 0
""")


def test_dropped_maps_give_way_to_allocations(run):
    """An allocation that needs the memory of dropped maps gets it: the same
    engine's, another slot's and another engine's."""
    run("""
a, b = engine(), engine()
a.set_receptor(1, R, gd)
before = fake.fake_live()
a.build_grids(0, HEAVY)
maps = fake.fake_live() - before
for user, rid in ((a, 1), (b, 0)):
    a.set_receptor(0, R, gd)  # drops slot 0's maps
    fake.fake_limit(fake.fake_live() + maps // 4)
    assert status(user.build_grids, rid, HEAVY) == sb.SG_OK
    fake.fake_limit(8 << 30)
    user.set_tables(T)
    a.build_grids(0, HEAVY)
""")


def test_a_failed_change_leaves_nothing_half_set(run):
    """After an allocation failed in sg_set_receptor or sg_set_tables, calls that
    would use the receptor or the tables are refused; after one in
    sg_set_user_grid the receptor has no grid.  Nothing runs on freed memory."""
    run("""
x = W.random_confs(m, gd, 2, 1)
big = W.receptor(9000)
e = engine()
uses = (lambda: e.bfgs(0, m, x), lambda: e.eval(0, m, x), lambda: e.minimize(0, [m], [0, 0], x),
        lambda: e.score(0, [m], [0, 0], x), lambda: e.build_grids(0, [2]))
def refused():
    n = fake.fake_launches(b"")
    assert all(status(f) == sb.SG_ERR_ARG for f in uses) and fake.fake_launches(b"") == n
def after_failures(change, check, least):
    failed, room = 0, 0
    while True:
        fake.fake_limit(fake.fake_live() + room)
        rc = status(change)
        fake.fake_limit(8 << 30)
        if rc == sb.SG_OK: break
        assert rc == sb.SG_ERR_NOMEM
        check()
        failed += 1
        room += 256 << 10
    assert failed >= least, failed
    assert all(status(f) == sb.SG_OK for f in uses), [status(f) for f in uses]
after_failures(lambda: e.set_receptor(0, big, W.box(30.0)), refused, 2)
def bare():  # the receptor without maps, so that none give way
    e.set_receptor(0, R, gd)
    uses[2]()
bare()
after_failures(lambda: e.set_tables(W.tables("ad4_scoring")), refused, 2)
small, larger = W.box(6.0), W.box(12.0)
bare()
e.set_user_grid(0, small, np.zeros(sb.grid_points(small)))
def no_grid(): assert fake.fake_dangling() == 0
no_grid()
after_failures(lambda: e.set_user_grid(0, larger, np.zeros(sb.grid_points(larger))), no_grid, 1)
""")


def test_a_failed_map_build_keeps_no_memory(run):
    """Memory taken for maps whose build then fails is given back."""
    run("""
e = engine()
bare = fake.fake_live()
e.build_grids(0, HEAVY)
maps = fake.fake_live() - bare
e.set_receptor(0, R, gd)
e.minimize(0, [m], [0], W.random_confs(m, gd, 1, 1))  # without maps again
bare = fake.fake_live()
fake.fake_limit(bare + maps + (64 << 10))  # room for the maps, not for the table that they are built from
for k in range(3):
    assert status(e.build_grids, 0, HEAVY) == sb.SG_ERR_NOMEM
    assert fake.fake_live() - bare < 1 << 20, k
fake.fake_limit(8 << 30)
assert status(e.build_grids, 0, HEAVY) == sb.SG_OK
""")


@pytest.mark.parametrize("call", ["score", "minimize", "dock", "dock_batch", "eval", "bfgs", "set_receptor", "build_grids",
                                  "create", "autotune"])
def test_host_allocation_failures_are_statuses(run, call):
    """The nth host allocation of a call fails, for every n: the call returns
    SG_ERR_NOMEM (or does without), the process goes on and the next call works."""
    run(f"call = {call!r}" + """
e = engine(sb.PREC_FP64 if call == "dock" else sb.PREC_FP32)
few = 64 if call == "score" else 3  # 64 models are packed on several threads
ms = [W.ligand(10 + k % 7, k % 3, k) for k in range(few)]
x = [W.random_confs(q, gd, 1, 1)[0] for q in ms]
cs = max(q.conf_size for q in ms)
confs = np.array([np.pad(c, (0, cs - len(c))) for c in x])
pm, p = list(range(few)), ms[0].search_params()
c0, mt = ms[0].seed_chains(5, 2, gd)
f = {"score": lambda: e.score(0, ms, pm, confs), "minimize": lambda: e.minimize(0, ms, pm, confs),
     "dock": lambda: e.dock(0, ms[:1], [0, 0], c0, mt, p, steps=1),
     "dock_batch": lambda: e.dock_batch(0, ms, [sb.LigandJob(model=k, num_chains=2, num_steps=2, maxiters=0, seed=1,
                                                             ligand_key=k) for k in pm], p),
     "eval": lambda: e.eval(0, ms[0], x[:1]), "bfgs": lambda: e.bfgs(0, ms[0], x[:1]),
     "set_receptor": lambda: e.set_receptor(0, R, gd), "create": lambda: sb.Engine(0, sb.PREC_FP32).close(),
     "autotune": lambda: e.autotune(0, ms, [sb.LigandJob(model=0, num_chains=2, num_steps=2, maxiters=0, seed=1,
                                                         ligand_key=0)], p, 1.0),
     "build_grids": lambda: (e.set_receptor(0, R, gd), e.build_grids(0, HEAVY))}[call]
assert status(f) == sb.SG_OK
n, failed = 0, 0
while True:
    n += 1
    fake.fake_fail_new(n)
    rc = status(f)
    if not fake.fake_new_fired(): break
    assert rc in (sb.SG_OK, sb.SG_ERR_NOMEM), rc
    failed += rc == sb.SG_ERR_NOMEM
    if call in ("set_receptor", "build_grids"): e.set_receptor(0, R, gd)
    if n % 16 == 0: assert status(f) == sb.SG_OK
assert failed > (1 if call == "create" else 10) and status(f) == sb.SG_OK
""")


def test_engines_on_threads_pin_memory_once(run):
    """Calls on eight engines at once pin one ring of memory each and keep it."""
    run("""
es = [engine() for _ in range(8)]
x = W.random_confs(m, gd, 4, 1)
for e in es: e.eval(0, m, x)
def at_once():
    fake.fake_sync_ms(40)  # every call lasts until all have begun
    ts = [threading.Thread(target=e.eval, args=(0, m, x)) for e in es]
    for t in ts: t.start()
    for t in ts: t.join()
    fake.fake_sync_ms(0)
before = fake.fake_host_allocs()
for k in range(4): at_once()
assert fake.fake_host_allocs() - before <= 8, fake.fake_host_allocs() - before
""")


def test_threads_do_not_lower_a_kernels_shared_memory(run):
    """Two engines launch the same kernel at once, the one that needs less
    shared memory a little later: the limit ends at the larger need."""
    run("""
es = [engine(sb.PREC_FP64), engine(sb.PREC_FP64)]
ms = [W.ligand(80, 20, 7), W.ligand(60, 12, 3)]  # both above the 48 KB that need no limit
for kernel, f in ((b"k_score64", lambda e, q: e.score(0, [q], [0], W.random_confs(q, gd, 1, 1))),
                  (b"k_refine64", lambda e, q: e.minimize(0, [q], [0], W.random_confs(q, gd, 1, 1)))):
    fake.fake_attr_ms(200)
    ts = [threading.Thread(target=f, args=a) for a in zip(es, ms)]
    ts[0].start()
    threading.Event().wait(0.1)
    ts[1].start()
    for t in ts: t.join()
    fake.fake_attr_ms(0)
    both = fake.fake_max_dynamic(kernel)
    f(es[0], ms[0])  # raises it again, had it been lowered
    assert both == fake.fake_max_dynamic(kernel) > 49152
""")


def test_launch_shapes_of_local_optimisations(run):
    """Warps per conf of the plain path's local optimisation, by the number of
    confs and of the model's pairs: one warp for many confs of small models."""
    run("""
e = engine(sb.PREC_FP64)
def warps(lig, n):
    q = W.ligand(*lig)
    x = np.repeat(W.random_confs(q, gd, 1, 1), n, 0)
    before = [fake.fake_launches(b"k_bfgs64ILi%dE" % w) for w in (1, 4, 8)]
    e.bfgs(0, q, x)
    return [w for w, k in zip((1, 4, 8), before) if fake.fake_launches(b"k_bfgs64ILi%dE" % w) != k]
SMALL, MIDDLE, LARGE = (10, 0, 4), (24, 5, 11), (36, 8, 5)
for lig, n, w in ((SMALL, 1, 8), (SMALL, 296, 8), (SMALL, 297, 4), (SMALL, 592, 4), (SMALL, 593, 1), (SMALL, 20000, 1),
                  (MIDDLE, 296, 8), (MIDDLE, 1184, 4), (MIDDLE, 2400, 1), (MIDDLE, 20000, 1), (LARGE, 296, 8),
                  (LARGE, 297, 4), (LARGE, 20000, 4), ((116, 30, 5), 2, 1)):
    assert warps(lig, n) == [w], (lig, n, w, warps(lig, n))
""")


def test_launch_shapes_of_refinements(run):
    """Warps per pose of the refinements: 8, but 4 for many poses of models with
    hardly any pairs."""
    run("""
e = engine(sb.PREC_FP64)
def warps(lig, n, call):
    q = W.ligand(*lig)
    x = np.repeat(W.random_confs(q, gd, 1, 1), n, 0)
    before = [fake.fake_launches(b"k_refine64ILi%dE" % w) for w in (1, 4, 8)]
    getattr(e, call)(0, [q], [0] * n, x)
    return [w for w, k in zip((1, 4, 8), before) if fake.fake_launches(b"k_refine64ILi%dE" % w) != k]
for call in ("refine", "minimize"):
    for lig, n, w in (((10, 0, 4), 296, 8), ((10, 0, 4), 297, 4), ((16, 2, 6), 5000, 4), ((24, 5, 11), 5000, 8),
                      ((50, 12, 3), 5000, 8), ((116, 30, 5), 2, 1)):
        assert warps(lig, n, call) == [w], (lig, n, w, warps(lig, n, call))
""")


def test_launch_shapes_of_mixed_precision_optimisations(run):
    """Warps per conf of the FP32 local optimisation (with the occupancies of
    128 registers a thread): 8 while all confs are resident, 4 up to 2.2 resident
    batches and fewer the fewer pairs there are, then one; 8 further where shared
    memory leaves no more room for 4."""
    run("""
e = engine()
def warps(lig, n):
    q = W.ligand(*lig)
    x = np.repeat(W.random_confs(q, gd, 1, 1), n, 0)
    before = fake.fake_launches(b"k_bfgs32_wide")
    e.bfgs(0, q, x)
    return fake.fake_threads(b"k_bfgs32_wide") // 32 if fake.fake_launches(b"k_bfgs32_wide") != before else 1
NONE, FEW, MANY, LARGE = (10, 0, 4), (16, 2, 6), (50, 12, 3), (80, 20, 7)  # 0, 61, 985 and 2,705 pairs
for lig, n, w in ((NONE, 1, 8), (NONE, 296, 8), (NONE, 592, 4), (NONE, 593, 1), (FEW, 297, 4), (FEW, 772, 4),
                  (FEW, 773, 1), (MANY, 296, 8), (MANY, 297, 4), (MANY, 1302, 4), (MANY, 1303, 1), (LARGE, 297, 8),
                  (LARGE, 5920, 8), (LARGE, 5921, 1)):
    assert warps(lig, n) == w, (lig, n, w, warps(lig, n))
""")


def test_batches_at_the_fixed_scratch_arrays_limit(run):
    """The largest batches that sg_dock_batch32_noalloc has taken still fit its
    8 MiB (3,757 ligands of 10 atoms, 209 of 24 with 8 chains of 9 places), the
    next larger ones do not."""
    run("""
e = engine()
def fits(lig, models, chains, places):
    q = W.ligand(*lig)
    e.build_grids(0, sorted({t for t in q.types() if 1 < t < 27}))
    p = q.search_params()
    p.num_saved_mins = places
    jobs = [sb.LigandJob(model=k, num_chains=chains, num_steps=1, maxiters=0, seed=1, ligand_key=k) for k in range(models)]
    try:
        e.dock_batch_noalloc(0, [q] * models, jobs, p)
    except sb.SminaError as x:  # (no kernel has written the results)
        return "corrupt" in str(x)
    return True
for lig, models, chains, places in (((10, 0, 4), 3757, 1, 1), ((24, 5, 11), 209, 8, 9), ((50, 12, 3), 219, 1, 1)):
    assert fits(lig, models, chains, places) and not fits(lig, models + 1, chains, places), lig
""")


def test_calls_do_without_pinned_memory(run):
    """Where no memory can be pinned, engines are created and calls copy all the same."""
    run("""
fake.fake_no_pinned(1)
e = engine()
x = W.random_confs(m, gd, 30000, 1)
assert status(e.eval, 0, m, x) == sb.SG_OK and fake.fake_host_allocs() == 0
c, _ = e.bfgs(0, m, x)  # (no kernel changes them: out and back)
assert np.array_equal(c, x)
fake.fake_no_pinned(0)
assert status(e.eval, 0, m, x) == sb.SG_OK and fake.fake_host_allocs() == 1
""")
