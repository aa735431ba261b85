"""Chains on several warps each (batches that leave warps idle) against the
search of one warp per chain, bit for bit: batches whose chains get 8 and 4 warps
on a B200 (296 and 592 resident blocks) and some past them, a model without
pairs, flexible residues, and charge-dependent tables; and local optimisations
on several warps against one."""
import numpy as np
import pytest

import smina_b200 as sb
import workloads as W

pytestmark = pytest.mark.gpu

VINA, AD4 = "vina", "ad4_scoring"
CASES = [
    (VINA, [(24, 5, 11)], 1, False), (VINA, [(24, 5, 11), (50, 12, 3), (10, 0, 4)], 3, False),
    (VINA, [(14, 3, 2)], 400, False), (VINA, [(14, 3, 2), (11, 0, 7)], 450, False), (VINA, [(12, 2, 2)], 1300, False),
    (VINA, [(20, 4, 5)], 4, True), (AD4, [(24, 5, 11)], 5, False),
]


@pytest.mark.parametrize("scoring,ligs,chains,flex", CASES)
def test_wide_chains_equal_one_warp(scoring, ligs, chains, flex):
    gd = W.box(26.0)
    eng = sb.Engine(0, sb.PREC_FP32)
    eng.set_tables(W.tables(scoring))
    if scoring == AD4:
        eng.set_receptor(0, W.charged_receptor(1500, 3, 2), gd)
        models = [W.charged_ligand(*lig, 1) for lig in ligs]
    else:
        eng.set_receptor(0, W.receptor(1500, 3), gd)
        fx = sb.make_flex_pdbqt(3, 42, W.CENTER) if flex else None
        models = [sb.Model(sb.make_ligand_pdbqt(*lig, W.CENTER), fx) for lig in ligs]
    jobs = [sb.LigandJob(model=k, num_chains=chains, num_steps=6, maxiters=0, seed=9, ligand_key=k)
            for k in range(len(models))]
    p = models[0].search_params()
    wide = eng.dock_batch(0, models, jobs, p, refine=False)
    lookups = eng.batch_stats()["pair_lookups"]
    eng.set_chains_per_block(4)  # one warp per chain
    one = eng.dock_batch(0, models, jobs, p, refine=False)
    assert eng.batch_stats()["pair_lookups"] == lookups
    for a, b in zip(wide, one):
        assert a["evals"] == b["evals"] > 0 and len(a["e"]) > 0
        for k in ("e", "conf", "coords"):
            assert np.array_equal(a[k], b[k]), k
    eng.close()


@pytest.mark.parametrize("scoring,lig,flex,prec", [
    (VINA, (10, 0, 4), False, sb.PREC_FP32), (VINA, (24, 5, 11), False, sb.PREC_FP32),
    (VINA, (50, 12, 3), False, sb.PREC_FP32_H16), (VINA, (20, 4, 5), True, sb.PREC_FP32),
    (AD4, (24, 5, 11), False, sb.PREC_FP32)])
def test_wide_optimisations_equal_one_warp(scoring, lig, flex, prec):
    """sg_bfgs: a conf's bits do not depend on the number of confs of the call,
    which decides between 8 warps, 4 and one per conf (test_host_failures.py)."""
    gd = W.box(26.0)
    eng = sb.Engine(0, prec)
    eng.set_tables(W.tables(scoring))
    eng.set_receptor(0, W.charged_receptor(1500, 3, 2) if scoring == AD4 else W.receptor(1500, 3), gd)
    fx = sb.make_flex_pdbqt(3, 42, W.CENTER) if flex else None
    m = W.charged_ligand(*lig, 1) if scoring == AD4 else sb.Model(sb.make_ligand_pdbqt(*lig, W.CENTER), fx)
    confs = W.random_confs(m, gd, 1400, 5)
    one = eng.bfgs(0, m, confs)
    assert np.isfinite(one[1]).all() and (one[0] != confs).any()
    for size in (592, 250, 1):
        last = 8 if size == 1 else len(confs)
        parts = [eng.bfgs(0, m, confs[k:min(k + size, last)]) for k in range(0, last, size)]
        assert np.array_equal(np.concatenate([c for c, _ in parts]), one[0][:last]), size
        assert np.array_equal(np.concatenate([e for _, e in parts]), one[1][:last]), size
    eng.close()


# ligands with their chains -> warps of the blocks, ligands that get them, and chains
# per block (148 SMs; two resident 8-warp or four 4-warp blocks on each)
SMALL, MIDDLE, LARGE = (12, 2, 2), (24, 5, 11), (50, 12, 3)
PLANS = [([(MIDDLE, 8)], (8, 1, 1)), ([(MIDDLE, 500)], (4, 1, 1)), ([(SMALL, 1300)], (0, 0, 1)),
         ([(LARGE, 20), (MIDDLE, 100), (SMALL, 900)], (8, 1, 8)),
         ([(LARGE, 300), (MIDDLE, 300), (SMALL, 600)], (4, 1, 4))]


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("ligs,plan", PLANS)
def test_each_plan_equals_one_warp(ligs, plan, early):
    """Blocks for all chains, for none and for the largest ligand beside the
    others' warps, in one search and in phases that resume (early stop, which
    here stops no ligand): the plan, and the bits of one warp per chain."""
    eng = sb.Engine(0, sb.PREC_FP32)
    eng.set_tables(W.tables())
    eng.set_receptor(0, W.receptor(1500, 3), W.box(26.0))
    models = [W.ligand(*lig) for lig, _ in ligs]
    jobs = [sb.LigandJob(model=k, num_chains=n, num_steps=6, maxiters=0, seed=9, ligand_key=k)
            for k, (_, n) in enumerate(ligs)]
    p = models[0].search_params()
    if early:
        eng.set_early_stop(checkpoints=3, first=1, fraction=1.0, eps=0.0)
    runs = []
    for shape in (0, 8):
        eng.set_chains_per_block(shape)
        r = eng.dock_batch(0, models, jobs, p, refine=False)
        runs.append((r, eng.batch_stats()))
    (wide, sw), (one, so) = runs
    assert (sw["block_warps"], sw["block_ligands"], sw["chains_per_block"]) == plan
    assert (so["block_warps"], so["block_ligands"], so["chains_per_block"]) == (0, 0, 8)
    assert sw["pair_lookups"] == so["pair_lookups"] > 0 and sw["grid_lookups"] == so["grid_lookups"] > 0
    for a, b in zip(wide, one):
        assert a["evals"] == b["evals"] > 0 and len(a["e"]) > 0
        for k in ("e", "conf", "coords"):
            assert np.array_equal(a[k], b[k]), k
    eng.close()


def test_autotune_keeps_the_automatic_launch_where_it_is_fastest():
    """A lone ligand's chains are fastest on a block each (50 heavy atoms: about
    half the time of one warp per chain), which is what sg_dock_batch32 does by
    itself: tuning must not turn that off."""
    eng = sb.Engine(0, sb.PREC_FP32)
    eng.set_tables(W.tables())
    eng.set_receptor(0, W.receptor(1500, 3), W.box(26.0))
    m = W.ligand(*LARGE)
    jobs = [sb.LigandJob(model=0, num_chains=8, num_steps=40, maxiters=0, seed=9, ligand_key=1)]
    p = m.search_params()
    chosen, rates = eng.autotune(0, [m], jobs, p, step_fraction=0.5)
    assert chosen == 1 and rates[1] == max(rates.values())
    tuned = eng.dock_batch(0, [m], jobs, p, refine=False)
    assert eng.batch_stats()["block_warps"] == 8
    eng.set_chains_per_block(1)
    one = eng.dock_batch(0, [m], jobs, p, refine=False)
    assert eng.batch_stats()["block_warps"] == 0 and np.array_equal(tuned[0]["conf"], one[0]["conf"])
    eng.close()
