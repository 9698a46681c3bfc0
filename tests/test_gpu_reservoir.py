"""The class-weighted sampler's parallel reservoir against the oracle at the edges of its
kernels: class counts around a lane each, 32 and more, segments and rows of odd lengths,
images above the bitmap's size, buckets that never fill, empty and absent classes.  Equal
sample lists."""
import numpy as np
import pytest

import padenti_gb300 as pg


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1, 2, 15, 16, 31, 32, 33, 64, 255])
@pytest.mark.parametrize("size", [(1, 1), (31, 1), (37, 29), (128, 4), (512, 3), (161, 121)])
def test_class_counts_and_sizes(K, size):
    import oracle_bind as ob

    w, h = size
    rng = np.random.default_rng(K * 1000 + w)
    px = [rng.integers(0, 5000, (h, w)).astype(np.uint16) for _ in range(3)]
    lb = [rng.integers(0, K + 1, (h, w)).astype(np.uint8) for _ in range(3)]
    lb[1][:] = np.where(rng.random((h, w)) < 0.97, 1, lb[1])  # one class nearly everywhere
    lb[2][:] = 0  # nothing labelled
    s = pg.ClassWeightedImageSampler(300, K, seed=5)
    for got, p, l in zip(s.sample_batch(px, lb), px, lb):
        assert np.array_equal(got, ob.sample_class_weighted(p, l, 300, K, None, 5))


@pytest.mark.gpu
def test_weights_and_mixed_sizes():
    """Zero and large weights, and images of different sizes in one batch."""
    import oracle_bind as ob

    rng = np.random.default_rng(9)
    K = 5
    sizes = [(640, 480), (3, 7), (700, 513), (160, 120)]
    px = [rng.integers(0, 5000, (h, w)).astype(np.uint16) for w, h in sizes]
    lb = [np.minimum(rng.integers(0, 9, (h, w)), K).astype(np.uint8) for w, h in sizes]
    lb[0][lb[0] == 2] = 0  # an absent class
    wts = np.array([0.0, 0.5, 3.0, 0.01, 1.0], np.float32)
    s = pg.ClassWeightedImageSampler(900, K, wts, seed=77)
    for got, p, l in zip(s.sample_batch(px, lb), px, lb):
        assert np.array_equal(got, ob.sample_class_weighted(p, l, 900, K, wts, 77))


@pytest.mark.gpu
def test_image_above_the_bitmap():
    import oracle_bind as ob

    rng = np.random.default_rng(3)
    px = rng.integers(0, 5000, (1025, 1030)).astype(np.uint16)  # 2^20 pixels and more
    lb = rng.integers(0, 4, px.shape).astype(np.uint8)
    s = pg.ClassWeightedImageSampler(1000, 3, seed=1)
    assert np.array_equal(s.sample(px, lb), ob.sample_class_weighted(px, lb, 1000, 3, None, 1))
