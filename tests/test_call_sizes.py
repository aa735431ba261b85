"""What a call returns for an item does not depend on the call's other items, on
what the engine held before, or on other engines' calls: batches that take other
launch shapes and more than one piece of the copies, maps of many types built at
once, receptors replaced in one place, engines on threads.  All bit for bit."""
import threading

import numpy as np
import pytest

import smina_b200 as sb
import workloads as W

pytestmark = pytest.mark.gpu

GD = W.box(26.0)


def engine(prec, scoring="vina", receptor=None, gd=GD):
    e = sb.Engine(0, prec)
    e.set_tables(W.tables(scoring))
    e.set_receptor(0, receptor or W.receptor(1500, 3), gd)
    return e


def same(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    assert a.shape == b.shape and a.tobytes() == b.tobytes()


@pytest.mark.parametrize("prec,threads,n,part", [
    (sb.PREC_FP32, 32, 1500, 100), (sb.PREC_FP32, 64, 1500, 100), (sb.PREC_FP32, 128, 1500, 100),
    (sb.PREC_FP32_H16, 32, 297, 33), (sb.PREC_FP32, 32, 20000, 4000), (sb.PREC_FP64, 32, 700, 200),
    (sb.PREC_FP64, 32, 6000, 250)])
def test_evaluations(prec, threads, n, part):
    """FP32 blocks of several confs from two per SM on, FP64 blocks that loop past
    four per SM; 20,000 confs are 2 MB each way, four times a piece of the copies."""
    e = engine(prec)
    e.set_threads_per_chain(threads)
    m = W.ligand(24, 5, 11)
    x = W.random_confs(m, GD, n, 5)
    whole = e.eval(0, m, x, coords=True)
    parts = [e.eval(0, m, x[k:k + part], coords=True) for k in range(0, n, part)]
    for k in range(3):
        same(whole[k], np.concatenate([p[k] for p in parts]))
    if prec == sb.PREC_FP64:
        whole = e.eval_direct(0, m, x)
        parts = [e.eval_direct(0, m, x[k:k + part]) for k in range(0, n, part)]
        for k in range(2):
            same(whole[k], np.concatenate([p[k] for p in parts]))
    e.close()


@pytest.mark.parametrize("scoring", ["vina", "ad4_scoring"])
@pytest.mark.parametrize("count", [1, 4, 5, 8, 9, 16, 17, 25])
def test_maps_of_many_types(scoring, count):
    """1 to 25 types at once (4, 8, 16 and 32 lanes a point) against one by one."""
    charged = scoring != "vina"
    rec = W.charged_receptor(1500, 3, 2) if charged else W.receptor(1500, 3)
    gd = W.box(12.0)
    many, single = engine(sb.PREC_FP64, scoring, rec, gd), engine(sb.PREC_FP64, scoring, rec, gd)
    types = list(range(2, 2 + count))
    many.build_grids(0, types)
    for t in types:
        single.build_grids(0, [t])
        a, b = many.grid(0, t, gd, charged), single.grid(0, t, gd, charged)
        same(a[0], b[0])
        if charged:
            same(a[1], b[1])
    many.close()
    single.close()


@pytest.mark.parametrize("prec", [sb.PREC_FP64, sb.PREC_FP32, sb.PREC_FP32_H16])
def test_receptors_replaced_in_one_place(prec):
    """Larger, smaller and charged receptors, other boxes, scoring and user grids
    one after the other in one place, whose memory they reuse, against engines
    that hold one each."""
    m, q = W.ligand(24, 5, 11), W.charged_ligand(24, 5, 11)
    types = list(range(2, 18))
    ug = W.box(9.0)
    values = np.random.default_rng(2).normal(size=sb.grid_points(ug))
    steps = [("vina", W.receptor(1500, 3), 22.0, None), ("vina", W.receptor(3000, 7), 26.0, None),
             ("vina", W.receptor(800, 5), 18.0, None), ("vina", W.receptor(800, 5), 18.0, values),
             ("ad4_scoring", W.charged_receptor(1500, 3, 2), 20.0, None), ("vina", W.receptor(1500, 3), 22.0, values),
             ("vina", W.receptor(1500, 3), 30.0, None)]

    def results(e, scoring, size):
        lig, gd = q if scoring != "vina" else m, W.box(size)
        e.build_grids(0, types)
        x = W.random_confs(lig, gd, 40, 3)
        out = [e.grid(0, t, gd)[0] for t in (2, 9, 17)]
        out += list(e.eval(0, lig, x)) + list(e.bfgs(0, lig, x[:9], maxiters=4))
        return out + list(e.minimize(0, [lig], [0] * 9, x[:9], maxiters=2))

    e = sb.Engine(0, prec)
    for scoring, rec, size, grid in steps:
        f = sb.Engine(0, prec)
        for g in (e, f):
            g.set_tables(W.tables(scoring))
            g.set_receptor(0, rec, W.box(size))
            if grid is not None:
                g.set_user_grid(0, ug, grid)
        for a, b in zip(results(e, scoring, size), results(f, scoring, size)):
            same(a, b)
        f.close()
    e.close()


def test_engines_on_threads():
    """Six engines call at once, evaluations, refinements and searches mixed,
    larger and smaller models, while receptors are set."""
    ms = [W.ligand(24, 5, 11), W.ligand(50, 12, 3), W.ligand(10, 0, 4)]

    def work(e, k):
        m = ms[k % 3]
        x = W.random_confs(m, GD, 600, k)
        e.set_receptor(0, W.receptor(1500, 3), GD)
        out = list(e.eval(0, m, x)) + list(e.bfgs(0, m, x, maxiters=3)) + list(e.score(0, [m], [0] * 50, x[:50]))
        out += list(e.minimize(0, [m], [0] * 5, x[:5], maxiters=2))
        if k < 3:
            r = e.dock_batch(0, [m], [sb.LigandJob(model=0, num_chains=8, num_steps=5, maxiters=0, seed=1, ligand_key=k)],
                             m.search_params())
            out += [r[0]["e"], r[0]["conf"]]
        return out

    es = [engine(sb.PREC_FP32 if k < 3 else sb.PREC_FP64) for k in range(6)]
    alone = [work(e, k) for k, e in enumerate(es)]
    got = [[None] * 3 for _ in es]

    def run(k):
        for r in range(3):
            got[k][r] = work(es[k], k)

    ts = [threading.Thread(target=run, args=(k,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k in range(6):
        for r in range(3):
            for a, b in zip(got[k][r], alone[k]):
                same(a, b)
    for e in es:
        e.close()
