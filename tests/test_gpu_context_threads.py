"""Contexts used from separate threads at once, with calls that take different amounts of
shared memory of the same kernels: no launch is refused, and every result is the one of a
thread alone."""
import threading

import numpy as np
import pytest

import padenti_gb300 as pg
from test_gpu_predict_forms import _random_tree
from test_gpu_rank_form import _depth_set


def _run(works, times):
    """Each work `times` times in its own thread; the results that differ from the first, and errors."""
    bad = []

    def loop(work):
        try:
            first = work()
            for _ in range(times):
                if not all(np.array_equal(a, b) for a, b in zip(first, work())):
                    bad.append("differs")
        except Exception as e:  # noqa: BLE001
            bad.append(repr(e))

    threads = [threading.Thread(target=loop, args=(w,)) for w in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return bad


def _training(K, T, thr):
    ts = _depth_set(51 + K, 6, 80, 60, K, 400)
    cfg = pg.ForestConfig("depth_diff2", K)
    tp = pg.TreeTrainerParameters(90, T, [-60000] * 4, [60000] * 4, -thr, thr, 5)
    tr = pg.TreeTrainer(cfg)
    tr.upload(ts)

    def work():
        t = pg.Tree(cfg, 2, 8)
        tr.train(t, ts, tp)
        return t.left_child, t.features, t.thresholds, t.posteriors

    return work


@pytest.mark.gpu
def test_training_of_different_shapes():
    assert _run([_training(3, 8, 500), _training(21, 60, 500), _training(9, 100, 900), _training(21, 40, 5000),
                 _training(3, 40, 5000)], 60) == []


@pytest.mark.gpu
def test_prediction_with_different_forests():
    rng = np.random.default_rng(4)
    cfg = pg.ForestConfig("depth_diff2", 3)
    img = rng.integers(500, 5000, (40, 60)).astype(np.uint16)

    def prediction(n_trees):
        clf = pg.Classifier(cfg)
        for _ in range(n_trees):
            clf << _random_tree(rng, cfg, 5, False)
        return lambda: (clf.predict(img),)

    assert _run([prediction(1), prediction(64), prediction(50)], 300) == []


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [pg.UniformImageSampler, pg.ClassWeightedImageSampler])
def test_samplers_of_different_sizes(kind):
    import torch

    from padenti_gb300 import _native as N

    rng = np.random.default_rng(5)

    def sampling(n_samples, w, h):
        img = torch.from_numpy(rng.integers(0, 256, (2, h, w)).astype(np.uint8)).cuda()
        lab = torch.from_numpy(rng.integers(0, 4, (2, h, w)).astype(np.uint8)).cuda()
        sm = kind(n_samples, *(() if kind is pg.UniformImageSampler else (3,)), seed=3)
        out = torch.zeros(2, sm.stride, dtype=torch.int32, device="cuda")
        cnt = torch.zeros(2, dtype=torch.int32, device="cuda")
        ctx, c = pg.Classifier(pg.ForestConfig("depth_diff2", 3)), sm._c(1)
        torch.cuda.synchronize()

        def work():
            N.check(N.lib().pd_sample_device(ctx.h, c, 2, img.data_ptr(), lab.data_ptr(), w, h, sm.stride, out.data_ptr(),
                                             cnt.data_ptr()))
            return out.cpu().numpy(), cnt.cpu().numpy()

        return work

    assert _run([sampling(100, 64, 48), sampling(16000, 1024, 640), sampling(6000, 800, 600)], 150) == []
