"""Histogram work items past the sizes that small training sets reach: 160000 samples with
sixteen candidate tiles on 152 SMs are cut into items of 4224 samples (full 32-sample batches,
several per warp, and a remainder that fills no whole round of the CTA's 16 warps), and nodes
of up to 4096 samples get their split in the small-node kernels of every class count.  Whole
trees against the oracle, tolerance 0."""
import pytest

import padenti_gb300 as pg
from test_gpu_rank_form import _depth_set, _tree_equal


@pytest.mark.gpu
@pytest.mark.parametrize("K,fuse_max", [(3, 4096), (8, 4096), (16, 4096), (21, 4096), (33, 4096), (3, 0), (21, 0)])
def test_long_items(K, fuse_max):
    ts = _depth_set(61 + K, 40, 160, 120, K, 4000)
    cfg = pg.ForestConfig("depth_diff2", K)
    tp = pg.TreeTrainerParameters(1000, 12, [-60000] * 4, [60000] * 4, -500, 500, 100)
    _tree_equal(cfg, ts, tp, 9, (("fuse_max", fuse_max),))
