"""The class-weighted sampler's draws, kept for a group of images at a time: batches cut into
several groups (images of one size and of different ones, groups that end on an image and
that do not) and an image larger than a group give the oracle's samples, on the device and the
host entry, and the next batch on the context too."""
import ctypes as C

import numpy as np
import pytest

import padenti_gb300 as pg
from padenti_gb300 import _native as N


@pytest.mark.gpu
@pytest.mark.parametrize("bytes_", [4096, 24000, 24576, 40000, 512 << 20])
def test_groups_of_draws(bytes_):
    import oracle_bind as ob
    import torch

    rng = np.random.default_rng(bytes_ % 97)
    K, n, w, h = 6, 7, 96, 64
    px = rng.integers(0, 5000, (n, h, w)).astype(np.uint16)
    lb = rng.integers(0, K + 1, (n, h, w)).astype(np.uint8)
    s = pg.ClassWeightedImageSampler(400, K, seed=11)
    ctx = pg.Classifier(pg.ForestConfig("depth_diff2", K))
    N.check(N.lib().pd_ctx_set_tuning(ctx.h, b"sample_group", bytes_))
    dpx, dlb = torch.from_numpy(px.view(np.int16)).cuda(), torch.from_numpy(lb).cuda()
    out = torch.zeros((n, s.stride), dtype=torch.int32, device="cuda")
    cnt = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    want = [ob.sample_class_weighted(p, l, 400, K, None, 11) for p, l in zip(px, lb)]
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        N.check(N.lib().pd_sample_device(ctx.h, C.byref(s._c(2)), n, dpx.data_ptr(), dlb.data_ptr(), w, h, s.stride,
                                         out.data_ptr(), cnt.data_ptr()))
        got, c = out.cpu().numpy().view(np.uint32), cnt.cpu().numpy()
        assert all(np.array_equal(got[i, :c[i]], want[i]) for i in range(n))
    # host images of different sizes
    sizes = [(96, 64), (17, 5), (200, 150), (33, 9), (96, 64)]
    ims = [rng.integers(0, 5000, (b, a)).astype(np.uint16) for a, b in sizes]
    lbs = [rng.integers(0, K + 1, (b, a)).astype(np.uint8) for a, b in sizes]
    P = C.c_void_p * len(sizes)
    U = C.c_uint32 * len(sizes)
    o = np.zeros((len(sizes), s.stride), np.uint32)
    c = np.zeros(len(sizes), np.uint32)
    N.check(N.lib().pd_sample(ctx.h, C.byref(s._c(2)), len(sizes), P(*[i.ctypes.data for i in ims]),
                              P(*[i.ctypes.data for i in lbs]), U(*[a for a, _ in sizes]), U(*[b for _, b in sizes]),
                              s.stride, o.ctypes.data, c.ctypes.data))
    for i in range(len(sizes)):
        assert np.array_equal(o[i, :c[i]], ob.sample_class_weighted(ims[i], lbs[i], 400, K, None, 11))


@pytest.mark.gpu
@pytest.mark.parametrize("K", [3, 20, 40])
def test_stretches_without_labels(K):
    """Images labelled in a few places only: segments (512 pixels) and pairs of them without a
    label, and ones with a single labelled pixel at either end."""
    import oracle_bind as ob

    rng = np.random.default_rng(K)
    w, h = 131, 100
    px = rng.integers(0, 5000, (4, h, w)).astype(np.uint16)
    lb = np.zeros((4, h * w), np.uint8)
    lb[0, [0, 511, 512, 1023, 1024, 5000, h * w - 1]] = [1, 2, 1, K, 2, 3, 1]
    lb[1, 4000:4700] = rng.integers(1, K + 1, 700)
    lb[2, h * w - 40:] = 2
    lb[3, rng.integers(0, h * w, 30)] = 3
    s = pg.ClassWeightedImageSampler(12, K, seed=2)
    lb = lb.reshape(4, h, w)
    for got, p, l in zip(s.sample_batch(list(px), list(lb)), px, lb):
        assert np.array_equal(got, ob.sample_class_weighted(p, l, 12, K, None, 2))
