"""The prediction kernels' two record forms (every node in the fast form, or one that is not)
and the padded posterior rows, against the oracle, at odd image sizes and class counts.
Posteriors and leaf ids, tolerance 0."""
import numpy as np
import pytest

import padenti_gb300 as pg

_BOUNDS = {"depth_diff2": 60000, "depth_diff1": 60, "channel_diff": 30}


def _random_tree(rng, cfg, depth, slow):
    """A random tree in heap order: leaves here and there, random posteriors."""
    t = pg.Tree(cfg, 0, depth)
    n, D = t.n_nodes, cfg.feat_dim
    b = _BOUNDS[cfg.plugin]
    t.features[:] = rng.integers(-b, b + 1, (n, D))
    if cfg.plugin == "channel_diff":
        t.features[:, :2] = rng.integers(0, 4, (n, 2))
    elif slow:
        t.features[rng.random(n) < 0.3, 0] = 30000 if cfg.plugin == "depth_diff1" else 3_000_000
    t.thresholds[:] = rng.integers(-300, 301, n)
    t.posteriors[:] = rng.random((n, cfg.n_classes), np.float32)
    t.left_child[0] = -1
    for i in range(n):
        if t.left_child[i] == -1 and 2 * i + 2 < n and (i < 7 or rng.random() < 0.8):
            t.left_child[i] = 2 * i + 1
            t.left_child[2 * i + 1] = t.left_child[2 * i + 2] = -1
    return t


@pytest.mark.gpu
@pytest.mark.parametrize("K,n_trees,size,masked", [(1, 1, (33, 9), False), (4, 2, (64, 40), True), (5, 3, (31, 17), False),
                                                   (9, 3, (95, 57), True), (21, 5, (1, 77), False), (64, 2, (40, 8), True)])
@pytest.mark.parametrize("slow", [False, True])
@pytest.mark.parametrize("plugin", ["depth_diff1", "depth_diff2", "channel_diff"])
def test_posteriors_and_leaves(plugin, slow, K, n_trees, size, masked):
    import oracle_bind as ob

    if slow and plugin == "channel_diff":
        pytest.skip("every channel-difference node takes the fast form")
    rng = np.random.default_rng(K * 100 + n_trees)
    w, h = size
    cfg = pg.ForestConfig(plugin, K)
    if plugin == "channel_diff":
        img = rng.integers(0, 256, (h, w, 3)).astype(np.uint8)
    else:
        img = rng.integers(500, 5000, (h, w)).astype(np.uint16)
        img[rng.random((h, w)) < 0.05] = 0
        img[rng.random((h, w)) < 0.05] = 45000  # negative as int16
    mask = (rng.random((h, w)) < 0.7).astype(np.uint8) if masked else None
    clf = pg.Classifier(cfg)
    trees = [_random_tree(rng, cfg, 4 + 2 * k, slow) for k in range(n_trees)]
    for t in trees:
        clf << t
    b = _BOUNDS[plugin]
    p = ob.params(cfg, pg.TreeTrainerParameters(64, 4, [-b] * cfg.feat_dim, [b] * cfg.feat_dim, -300, 300, 1))
    tt = [(t.depth, t.left_child, np.asarray(t.features, np.int32), np.asarray(t.thresholds, np.int32), t.posteriors)
          for t in trees]
    post = clf.predict(img, mask)
    ref = ob.predict_posterior(p, img, mask, tt, n_channels=cfg.n_channels)
    assert np.array_equal(post.view(np.uint32), ref.view(np.uint32))
    assert np.array_equal(clf.predict_batch([img], [mask])[0].view(np.uint32), ref.view(np.uint32))
    for k, t in enumerate(trees):
        leaf = ob.predict_leaf(p, img, mask, t.depth, t.left_child, tt[k][2], tt[k][3], n_channels=cfg.n_channels)
        assert np.array_equal(clf.predict_leaf(k, img, mask), leaf)
