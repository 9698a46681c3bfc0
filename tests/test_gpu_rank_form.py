"""The rank-table form of the histogram kernels (thresholds looked up, large nodes in chunks,
small nodes with the split fused by the number of classes present) against the oracle at the
edges of its dispatch, and the one-multiply-add offset rounding against the plugins' float
formula.  Whole trees are compared, tolerance 0."""
import numpy as np
import pytest

import padenti_gb300 as pg


def _fma_round(u, d):
    """x + fl-rounded offset of pd_plugins.cuh fast_coord: fl(u' fl(1/d) + M) - M.  The product
    and sum are exact enough in float64: no value lies within 2^-29 of a tie (checked)."""
    inv = (np.float32(1) / d.astype(np.float32)).astype(np.float64)
    q = (u + np.where(u < 0, -0.25, 0.25)) * inv
    assert np.all(np.abs(np.abs(q - np.floor(q)) - 0.5) > 2.0**-22)
    return np.rint(q).astype(np.int64)


def _float_round(u, d):
    q = (u.astype(np.float32) / d.astype(np.float32)).astype(np.float64)
    return np.trunc(q + np.copysign(0.5, q)).astype(np.int64)


def test_offset_rounding_every_depth():
    d = np.arange(1, 65536, dtype=np.int64)
    for k in (0, 1, 2, 3, 7, 37, 75, 1000):
        for delta in (-1, 0, 1):
            for u0 in ((2 * k + 1) * d // 2 + delta, k * d + delta):
                u = np.clip(u0, -(2**21), 2**21)
                for sign in (1, -1):
                    assert np.array_equal(_fma_round(sign * u, d), _float_round(sign * u, d))


def test_offset_rounding_random():
    rng = np.random.default_rng(1)
    u = rng.integers(-(2**21), 2**21 + 1, size=2_000_000)
    d = rng.integers(1, 65536, size=2_000_000)
    assert np.array_equal(_fma_round(u, d), _float_round(u, d))


def _tree_equal(cfg, ts, tp, depth, tuning=()):
    import oracle_bind as ob

    tr = pg.TreeTrainer(cfg)
    for name, value in tuning:
        tr.set_tuning(name, value)
    tree = pg.Tree(cfg, 3, depth)
    tr.train(tree, ts, tp)
    o = ob.train_tree(ob.params(cfg, tp), ob.OracleSet(ts, cfg), 3, depth, ts.priors)
    assert int((o["left_child"] >= 0).sum()) >= 3
    assert np.array_equal(tree.left_child, o["left_child"])
    assert np.array_equal(tree.features, o["features"])
    assert np.array_equal(tree.thresholds, o["thresholds"])
    assert np.array_equal(tree.posteriors.view(np.uint32), o["posteriors"].view(np.uint32))


def _depth_set(seed, n, w, h, K, samples, big=False):
    """Depth maps (K classes by vertical stripes on the objects) and their samples."""
    px, lb, _ = pg.synth_depth(seed, n, w, h, parts=1, min_ellipses=2, max_ellipses=5, samples_per_image=4)
    rng = np.random.default_rng(seed)
    x = np.arange(w)[None, None, :]
    lb = (1 + (lb.astype(np.int64) * 7 + x * K // w) % K).astype(np.uint8)
    if big:  # zero depths, and depths above 32767 (negative as int16)
        px = np.where(rng.random(px.shape) < 0.02, 0, px).astype(np.uint16)
        px = np.where(rng.random(px.shape) < 0.02, 40000, px).astype(np.uint16)
    sm = np.sort(rng.integers(0, w * h, (n, samples)).astype(np.uint32), axis=1)
    return pg.training_set(K, px, lb, sm)


@pytest.mark.gpu
@pytest.mark.parametrize("T,lo,hi", [
    (1, -500, 500), (31, -500, 500), (32, -300, 400), (33, -7, 8), (50, 0, 0), (64, -1023, 1022), (65, -1023, 1023),
    (20, -1023, 1024), (100, -60, 60),
])
def test_thresholds_and_ranges(T, lo, hi):
    """Threshold counts around a word, ranges with many duplicates, the widest table and the
    first range that goes back to the search."""
    ts = _depth_set(11, 6, 81, 61, 3, 400)
    cfg = pg.ForestConfig("depth_diff2", 3)
    tp = pg.TreeTrainerParameters(70, T, [-60000] * 4, [60000] * 4, lo, hi, 10)
    _tree_equal(cfg, ts, tp, 6)


@pytest.mark.gpu
@pytest.mark.parametrize("K,F", [(2, 1), (4, 63), (5, 64), (8, 65), (9, 128), (17, 70), (32, 33), (33, 70), (64, 20)])
def test_class_rows(K, F):
    """Every small-node kernel, nodes with more classes than the widest, one to three tiles."""
    ts = _depth_set(21 + K, 5, 96, 64, K, 500)
    cfg = pg.ForestConfig("depth_diff2", K)
    tp = pg.TreeTrainerParameters(F, 12, [-60000] * 4, [60000] * 4, -500, 500, 5)
    _tree_equal(cfg, ts, tp, 7)


@pytest.mark.gpu
@pytest.mark.parametrize("tuning", [(), (("fuse_max", 0),), (("chunk", 256), ("persist", 1)), (("hist_spi", 4),),
                                    (("hist_spi", 2), ("cand_order", 0))])
@pytest.mark.parametrize("plugin", ["depth_diff1", "depth_diff2", "channel_diff"])
def test_plugins_and_shapes(plugin, tuning):
    """Every built-in feature, chunked and fused, with samples whose centre depth is zero or
    negative as int16 (depth_diff1) and odd image sizes."""
    if plugin == "channel_diff":
        px, lb, sm = pg.synth_rgb(5, 6, 53, 47, n_classes=11, samples_per_image=700)
        ts = pg.training_set(11, px, lb, sm)
        tp = pg.TreeTrainerParameters(90, 30, [0, 0] + [-30] * 4, [3, 3] + [30] * 4, -255, 255, 6)
        _tree_equal(pg.ForestConfig(plugin, 11), ts, tp, 8, tuning)
        return
    ts = _depth_set(31, 6, 77, 59, 5, 700, big=True)
    D, b = (2, 60) if plugin == "depth_diff1" else (4, 60000)
    tp = pg.TreeTrainerParameters(90, 30, [-b] * D, [b] * D, -200, 200, 6)
    _tree_equal(pg.ForestConfig(plugin, 5), ts, tp, 8, tuning)


@pytest.mark.gpu
def test_pure_and_constant_nodes():
    """Nodes of one class, and images on which no candidate separates anything: the winner is
    the lowest index among equal gains."""
    K, n, w, h = 3, 3, 64, 48
    px = np.full((n, h, w), 1500, np.uint16)
    lb = np.ones((n, h, w), np.uint8)
    lb[:, :, w // 2:] = 2
    px[:, :, w // 2:] = 1500
    px[2, :, : w // 4] = 900
    rng = np.random.default_rng(3)
    sm = np.sort(rng.integers(0, w * h, (n, 300)).astype(np.uint32), axis=1)
    ts = pg.training_set(K, px, lb, sm)
    tp = pg.TreeTrainerParameters(66, 9, [-60000] * 4, [60000] * 4, -500, 500, 1)
    cfg = pg.ForestConfig("depth_diff2", K)
    _tree_equal(cfg, ts, tp, 5)
