"""The device merge of a ligand's chains against the host's, bit for bit: the
batched search merges on the device, its no-allocation twin on the host, from
the same chains.  One chain and many; one place, less and more places than a
group of poses (32, or 8 where the places are many), and the most there can be."""
import numpy as np
import pytest

import smina_b200 as sb
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lig,chains,places,steps", [
    ((10, 0, 4), 1, 1, 20), ((24, 5, 11), 33, 1, 10), ((24, 5, 11), 200, 9, 20), ((12, 2, 2), 100, 33, 60),
    ((12, 2, 2), 1500, 9, 8), ((10, 0, 4), 40, 130, 120), ((10, 0, 4), 25, 200, 300), ((10, 0, 4), 20, 1024, 400)])
def test_merge_equals_the_hosts(lig, chains, places, steps):
    eng = sb.Engine(0, sb.PREC_FP32)
    eng.set_tables(W.tables())
    eng.set_receptor(0, W.receptor(), W.box())
    m = W.ligand(*lig)
    eng.build_grids(0, sorted({t for t in m.types() if 1 < t < 27}))
    p = m.search_params()
    p.num_saved_mins = places
    jobs = [sb.LigandJob(model=0, num_chains=n, num_steps=steps, maxiters=0, seed=7 + n, ligand_key=3)
            for n in (chains, 1)]  # a second ligand whose chains follow
    host = eng.dock_batch_noalloc(0, [m], jobs, p)
    device = eng.dock_batch(0, [m], jobs, p, refine=False)
    for a, b in zip(device, host):
        assert len(a["e"]) == len(b["e"]) > 0 and a["evals"] == b["evals"]
        for k in ("e", "conf", "coords"):
            assert np.array_equal(a[k], b[k]), k
    assert places > 200 or len(device[0]["e"]) >= min(places, 20)  # the places are fought over
    eng.close()
