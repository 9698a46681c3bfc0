"""The histogram launches of a level -- large nodes, and small nodes by the classes present --
run side by side on streams of the context: levels that hold all of them, trained repeatedly
and by two contexts at once, against the oracle.  Tolerance 0."""
import threading

import numpy as np
import pytest

import padenti_gb300 as pg
from test_gpu_rank_form import _depth_set


@pytest.mark.gpu
@pytest.mark.parametrize("K,fuse_max,persist", [(20, 4096, 0), (20, 64, 0), (20, 4096, 1), (3, 4096, 0), (40, 4096, 0)])
def test_levels_of_several_launches(K, fuse_max, persist):
    import oracle_bind as ob

    ts = _depth_set(41, 8, 96, 72, K, 1500)
    cfg = pg.ForestConfig("depth_diff2", K)
    tp = pg.TreeTrainerParameters(90, 20, [-60000] * 4, [60000] * 4, -400, 400, 4)
    o = ob.train_tree(ob.params(cfg, tp), ob.OracleSet(ts, cfg), 2, 9, ts.priors)
    bad = []

    def run():
        tr = pg.TreeTrainer(cfg)
        tr.set_tuning("fuse_max", fuse_max)
        tr.set_tuning("persist", persist)
        for _ in range(4):
            t = pg.Tree(cfg, 2, 9)
            tr.train(t, ts, tp)
            ok = (np.array_equal(t.left_child, o["left_child"]) and np.array_equal(t.features, o["features"])
                  and np.array_equal(t.thresholds, o["thresholds"])
                  and np.array_equal(t.posteriors.view(np.uint32), o["posteriors"].view(np.uint32)))
            bad.append(not ok)

    threads = [threading.Thread(target=run) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(bad) == 8 and not any(bad)
