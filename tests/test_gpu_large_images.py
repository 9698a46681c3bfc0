"""Prediction of images whose sides do not fit 16 bits (or, for the two-probe depth feature,
the range in which its offsets are rounded by one multiply-add), with a forest all of whose
nodes take the fast form: posteriors, masks and leaf ids against the oracle, tolerance 0."""
import numpy as np
import pytest

import padenti_gb300 as pg
from test_gpu_predict_forms import _BOUNDS, _random_tree


@pytest.mark.gpu
@pytest.mark.parametrize("plugin,size", [
    ("depth_diff1", (65535, 3)), ("depth_diff1", (65536, 2)), ("depth_diff1", (70000, 3)), ("depth_diff1", (3, 70000)),
    ("depth_diff2", (70000, 3)), ("depth_diff2", (2**21, 1)), ("depth_diff2", (2**22 + 999, 1)),
    ("channel_diff", (70000, 3)),
])
def test_sides_past_the_fast_form(plugin, size):
    import oracle_bind as ob

    w, h = size
    rng = np.random.default_rng(w + 7 * h)
    K = 3
    cfg = pg.ForestConfig(plugin, K)
    if plugin == "channel_diff":
        img = rng.integers(0, 256, (h, w, 3)).astype(np.uint8)
    else:
        img = rng.integers(500, 5000, (h, w)).astype(np.uint16)
        img[rng.random((h, w)) < 0.05] = 0
    mask = (rng.random((h, w)) < 0.9).astype(np.uint8)
    trees = [_random_tree(rng, cfg, 6, False) for _ in range(2)]
    for t in trees:
        first = 2 if plugin == "channel_diff" else 0  # offsets that often stay inside a few rows or columns
        t.features[:, first::2] //= max(1, 60 // w)
        t.features[:, first + 1::2] //= max(1, 60 // h)
        t.thresholds //= 4
    b = _BOUNDS[plugin]
    p = ob.params(cfg, pg.TreeTrainerParameters(64, 4, [-b] * cfg.feat_dim, [b] * cfg.feat_dim, -300, 300, 1))
    tt = [(t.depth, t.left_child, np.asarray(t.features, np.int32), np.asarray(t.thresholds, np.int32), t.posteriors)
          for t in trees]
    clf = pg.Classifier(cfg)
    for t in trees:
        clf << t
    small = np.ascontiguousarray(img[:, :40])
    for im, mk in ((img, mask), (small, None), (img, None)):  # both forms of the records, in turn
        ref = ob.predict_posterior(p, im, mk, tt, n_channels=cfg.n_channels)
        assert np.array_equal(clf.predict(im, mk).view(np.uint32), ref.view(np.uint32))
        for k, t in enumerate(trees):
            leaf = ob.predict_leaf(p, im, mk, t.depth, t.left_child, tt[k][2], tt[k][3], n_channels=cfg.n_channels)
            assert np.array_equal(clf.predict_leaf(k, im, mk), leaf)
            assert len(np.unique(leaf[leaf > 0])) > 2
