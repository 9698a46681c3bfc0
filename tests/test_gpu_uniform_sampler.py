"""The uniform sampler's bucket sort and rank walk against the oracle: sample counts around the
CTA's width and the largest, few labelled pixels (many equal draws), one, none, and sizes
around the label vectors.  Equal sample lists."""
import numpy as np
import pytest

import padenti_gb300 as pg


@pytest.mark.gpu
@pytest.mark.parametrize("n_samples", [1, 2, 255, 256, 257, 2000, 16384])
@pytest.mark.parametrize("size", [(1, 1), (5, 3), (16, 1), (64, 16), (131, 97), (640, 480)])
def test_sample_counts_and_sizes(n_samples, size):
    import oracle_bind as ob

    w, h = size
    rng = np.random.default_rng(n_samples + w)
    px = [rng.integers(0, 5000, (h, w)).astype(np.uint16) for _ in range(5)]
    lb = [(rng.random((h, w)) < p).astype(np.uint8) * 200 for p in (1.1, 0.5, 0.02, 0.0, 0.9)]
    lb[2].reshape(-1)[-1] = 1  # few labelled pixels, the last among them
    lb[4].reshape(-1)[: (w * h) // 2] = 0
    s = pg.UniformImageSampler(n_samples, seed=12)
    for got, p, l in zip(s.sample_batch(px, lb), px, lb):
        assert np.array_equal(got, ob.sample_uniform(p, l, n_samples, 12))
