"""The plain path's launch shapes against the oracle, bit for bit: 8 warps per
item (few items), 4 warps (more than two items per SM), and one warp with
nothing staged (a model whose staged form exceeds an SM's shared memory while
its plain form fits), each through every kernel of the path."""
import numpy as np
import pytest

import smina_b200 as sb
import workloads as W
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu

# ligand (heavy, rotors, seed), items: 2 x 148 + 9 items leave the 8-warp shape;
# the last ligand's 5,996 pairs alone take 192 KB (the plain form 218 KB, the
# staged form 236 KB of the 232 KB an SM gives a block)
SHAPES = [((24, 5, 11), 3), ((17, 4, 2), 305), ((116, 30, 5), 2)]


def same(a, b, what):
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
    assert a.shape == b.shape and np.array_equal(a.view(np.uint64), b.view(np.uint64)), what


@pytest.mark.parametrize("lig,n", SHAPES)
def test_every_kernel_at_every_shape(lig, n):
    T, R = W.tables(), W.receptor(1500, 3)
    gd = W.box(26.0)
    m = W.ligand(*lig)
    if lig[0] > 100:
        assert 5900 <= m.desc.num_pairs <= 6400
    eng = sb.Engine(0, sb.PREC_FP64)
    eng.set_tables(T)
    eng.set_receptor(0, R, gd)
    orc = Oracle(T, R, gd, full_cells=True)
    confs = W.random_confs(m, gd, n, 5)
    for a, b in zip(eng.eval(0, m, confs), orc.eval(m, confs)):
        same(a, b, "eval")
    for a, b in zip(eng.eval_direct(0, m, confs), orc.eval_direct(m, confs)):
        same(a, b, "eval_direct")
    (c1, e1), (c0, e0) = eng.bfgs(0, m, confs, maxiters=3), orc.bfgs(m, confs, maxiters=3)
    same(c1, c0, "bfgs confs")
    same(e1, e0, "bfgs energies")
    pm = [0] * n
    for a, b in zip(eng.refine(0, [m], pm, confs, maxiters=2), orc.refine([m], pm, confs, maxiters=2)):
        same(a, b, "refine")
    for a, b in zip(eng.score(0, [m], pm, confs), orc.score([m], pm, confs)):
        same(a, b, "score")
    p = m.search_params()
    p.maxiters = 3
    c, mt = m.seed_chains(5, n, gd)
    b1, b0 = eng.dock(0, [m], pm, c, mt, p, steps=2), orc.dock([m], pm, c, mt, p, steps=2)
    assert (b1.count == b0.count).all()
    same(b1.e, b0.e, "chain energies")
    same(b1.coords, b0.coords, "chain poses")
    eng.close()


@pytest.mark.parametrize("lig,n", [((10, 0, 4), 593), ((24, 5, 11), 2000)])
def test_many_small_optimisations_equal_few(lig, n):
    """Past a few confs per SM small models get one warp per conf: the same bits
    as in calls of 4 and 8 warps per conf."""
    eng = sb.Engine(0, sb.PREC_FP64)
    eng.set_tables(W.tables())
    eng.set_receptor(0, W.receptor(1500, 3), W.box(26.0))
    m = W.ligand(*lig)
    confs = W.random_confs(m, W.box(26.0), n, 5)
    c1, e1 = eng.bfgs(0, m, confs)
    for size in (500, 250):  # 4 warps, 8 warps
        parts = [eng.bfgs(0, m, confs[k:k + size]) for k in range(0, n, size)]
        same(c1, np.concatenate([c for c, _ in parts]), "confs")
        same(e1, np.concatenate([e for _, e in parts]), "energies")
    eng.close()
