"""The measured workloads of padenti_gb300: training, prediction, pixel sampling and label
mapping through the package's public entry points (the Python classes, and the C ABI for
buffers that are already in device memory).

A case is a dict of plain values.  Images, labels, samples and forests are made on the GPU
from the seed alone; ``prepare`` hands over what a user's program holds before the call (a
trainer with its training set uploaded, a classifier with its forest, image buffers).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import padenti_gb300 as pg
from padenti_gb300 import _native as N

# image type, channels, feature dimension and bounds of the built-in features
_FEATURES = {
    "depth_diff2": dict(low=[-60000] * 4, up=[60000] * 4, thr=500),
    "depth_diff1": dict(low=[-60] * 2, up=[60] * 2, thr=200),
    "channel_diff": dict(low=[0, 0, -30, -30, -30, -30], up=[3, 3, 30, 30, 30, 30], thr=255),
}


def listed():
    return [
        # One tree of the small configuration: 64 depth maps of 160x120.  Each level is a
        # few hundred microseconds of kernels: launches, copies and waits count.
        dict(name="train-small", what="train", feature="depth_diff2", images=64, width=160, height=120, mixed=False,
             classes=3, samples=500, features=200, thresholds=20, depth=8, min_leaf=20),
        # One tree of the benchmark's forest on 640x480 depth maps (600 of its 2000 images):
        # the ordinary large training run.
        dict(name="train-depth", what="train", feature="depth_diff2", images=600, width=640, height=480, mixed=False,
             classes=9, samples=2000, features=2000, thresholds=50, depth=16, min_leaf=20),
        # Depth maps of three sizes in one set, down to depth 20: uneven frontiers of many
        # small nodes, and tree arrays of a million nodes.
        dict(name="train-mixed", what="train", feature="depth_diff2", images=240, width=640, height=480, mixed=True,
             classes=9, samples=2000, features=1000, thresholds=50, depth=20, min_leaf=20),
        # RGB images with 21 classes: 8-bit three-channel probes, wide histograms.
        dict(name="train-rgb", what="train", feature="channel_diff", images=200, width=320, height=240, mixed=False,
             classes=21, samples=2000, features=1000, thresholds=30, depth=18, min_leaf=10),
        # The one-offset feature with int16 responses, on images and candidate counts that
        # are no multiple of anything.
        dict(name="train-short", what="train", feature="depth_diff1", images=101, width=317, height=211, mixed=False,
             classes=3, samples=1333, features=777, thresholds=10, depth=10, min_leaf=133),
        # The smallest prediction: one host image with a mask, posteriors back on the host.
        dict(name="predict-one", what="predict", feature="depth_diff2", images=1, width=160, height=120, classes=3,
             trees=1, depth=8, mask=True),
        # Posteriors of a block of held-out images that is in device memory already.
        dict(name="predict-depth", what="predict_device", feature="depth_diff2", images=160, width=640, height=480,
             classes=9, trees=3, depth=16, mask=False),
        # The same for the RGB forest: five deeper trees, 21 planes out.
        dict(name="predict-rgb", what="predict_device", feature="channel_diff", images=100, width=320, height=240,
             classes=21, trees=5, depth=18, mask=False),
        # Serving: a batch of host images of three sizes in one call.
        dict(name="predict-batch", what="predict_batch", feature="depth_diff2", images=48, width=640, height=480,
             classes=9, trees=3, depth=16, mask=False),
        # 2000 pixels of each image, uniformly over its labelled pixels.
        dict(name="sample-uniform", what="sample", kind="uniform", images=500, width=640, height=480, classes=9,
             samples=2000),
        # The class-weighted reservoir over the same kind of images.
        dict(name="sample-weighted", what="sample", kind="class_weighted", images=500, width=640, height=480,
             classes=9, samples=2000),
        # Colour-coded label images to classes.
        dict(name="labels", what="labels", images=400, width=640, height=480, classes=9, channels=3),
    ]


def _spread(rng, lo, hi):
    """An integer in [lo, hi], spread over its logarithm where the range is wide."""
    if hi > 10 * lo:
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))
    return rng.randint(lo, hi)


def draw(rng):
    what = rng.choice(["train", "train", "train", "predict", "predict_device", "predict_device", "predict_batch",
                       "sample", "sample", "labels"])
    if what == "labels":
        return dict(what=what, images=_spread(rng, 1, 400), width=_spread(rng, 80, 640), height=_spread(rng, 60, 480),
                    classes=rng.randint(2, 40), channels=rng.choice([3, 4]))
    if what == "sample":
        # the device call takes images whose pixel count is a multiple of 16
        return dict(what=what, kind=rng.choice(["uniform", "class_weighted"]), images=_spread(rng, 1, 500),
                    width=16 * rng.randint(5, 40), height=_spread(rng, 60, 480), classes=rng.randint(2, 21),
                    samples=_spread(rng, 100, 2500))
    feature = rng.choice(["depth_diff2", "depth_diff2", "channel_diff"] + (["depth_diff1"] if what == "train" else []))
    classes = 21 if feature == "channel_diff" else 3 if feature == "depth_diff1" else rng.choice([3, 9])
    if what == "train":
        c = dict(what=what, feature=feature, images=_spread(rng, 16, 600), width=_spread(rng, 100, 640),
                 height=_spread(rng, 80, 480), mixed=rng.random() < 0.2, classes=classes, samples=_spread(rng, 300, 2000),
                 features=_spread(rng, 60, 2000), thresholds=rng.randint(8, 60 if classes < 21 else 40),
                 depth=rng.randint(6, 16), min_leaf=rng.randint(5, 40))
        while c["images"] * c["samples"] * c["features"] * c["depth"] > 3.5e10:
            c["images"] = max(16, c["images"] // 2)
            c["features"] = max(60, c["features"] * 3 // 4)
        return c
    images = {"predict": 1, "predict_device": _spread(rng, 1, 120), "predict_batch": _spread(rng, 2, 40)}[what]
    return dict(what=what, feature=feature, images=images, width=_spread(rng, 100, 640),
                height=_spread(rng, 80, 480), classes=classes, trees=rng.randint(1, 4), depth=rng.randint(6, 16),
                mask=rng.random() < 0.3)


# ------------------------------------------------------------------- inputs ----
_DEV = "cuda"


def _gen(seed):
    g = torch.Generator(device=_DEV)
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 12345)
    return g


def _u(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, device=_DEV) * (hi - lo) + lo


def _depth_images(g, n, w, h, classes):
    """Depth maps in millimetres (uint16 values in int32) and labels (class + 1): a noisy
    background plane, 2 to 5 ellipses split into classes - 1 angular sectors, and a few
    pixels without a reading (0)."""
    e = 5
    scale = w / 160.0
    count = torch.randint(2, e + 1, (n,), generator=g, device=_DEV)
    cx, cy = _u(g, 0.15 * w, 0.85 * w, n, e), _u(g, 0.15 * h, 0.85 * h, n, e)
    ax, ay = _u(g, 10 * scale, 40 * scale, n, e), _u(g, 10 * scale, 40 * scale, n, e)
    dist, plane = _u(g, 800, 2500, n, e), _u(g, 3000, 4000, n)
    y = torch.arange(h, device=_DEV, dtype=torch.float32).view(1, h, 1)
    x = torch.arange(w, device=_DEV, dtype=torch.float32).view(1, 1, w)
    depth = plane.view(n, 1, 1).expand(n, h, w).clone()
    label = torch.ones(n, h, w, dtype=torch.uint8, device=_DEV)
    for k in range(e):
        v = lambda a: a[:, k].view(n, 1, 1)  # noqa: E731
        dx, dy = (x - v(cx)) / v(ax), (y - v(cy)) / v(ay)
        inside = (dx * dx + dy * dy < 1) & (k < count).view(n, 1, 1)
        part = ((torch.atan2(dy, dx) / (2 * math.pi) + 0.5) * (classes - 1)).floor().clamp(0, classes - 2)
        depth = torch.where(inside, v(dist).expand_as(depth), depth)
        label = torch.where(inside, (part + 2).to(torch.uint8), label)
    depth = (depth + 5 * torch.randn(n, h, w, generator=g, device=_DEV)).round().clamp(500, 9999)
    depth = torch.where(torch.rand(n, h, w, generator=g, device=_DEV) < 0.003, torch.zeros_like(depth), depth)
    return depth.to(torch.int32), label


def _palette(classes):
    r = np.random.RandomState(77)
    return r.randint(20, 236, (classes, 3)).astype(np.int64) // 3 * 3 + np.arange(classes)[:, None] % 3


def _rgb_images(g, n, w, h, classes):
    """Voronoi images [n][h][w][3] (uint8 values in int32) with texture noise, and labels."""
    cells = 20
    count = torch.randint(8, cells + 1, (n,), generator=g, device=_DEV)
    px, py = _u(g, 0, w, n, cells), _u(g, 0, h, n, cells)
    cls = torch.randint(0, classes, (n, cells), generator=g, device=_DEV)
    y = torch.arange(h, device=_DEV, dtype=torch.float32).view(1, h, 1)
    x = torch.arange(w, device=_DEV, dtype=torch.float32).view(1, 1, w)
    best = torch.full((n, h, w), 1e30, device=_DEV)
    label = torch.zeros(n, h, w, dtype=torch.int64, device=_DEV)
    for k in range(cells):
        d = (x - px[:, k].view(n, 1, 1)) ** 2 + (y - py[:, k].view(n, 1, 1)) ** 2
        near = (d < best) & (k < count).view(n, 1, 1)
        best = torch.where(near, d, best)
        label = torch.where(near, cls[:, k].view(n, 1, 1), label)
    colour = torch.from_numpy(_palette(classes)).to(_DEV)[label]
    noise = torch.randint(-20, 21, colour.shape, generator=g, device=_DEV)
    return (colour + noise).clamp(0, 255).to(torch.int32), (label + 1).to(torch.uint8)


def _images(g, feature, n, w, h, classes):
    """n images and labels, made a few at a time so that the float temporaries stay small."""
    make = _rgb_images if feature == "channel_diff" else _depth_images
    step = max(1, (1 << 24) // (w * h))
    parts = [make(g, min(step, n - i), w, h, classes) for i in range(0, n, step)]
    dt = torch.uint8 if feature == "channel_diff" else torch.int16  # uint16 depths are below 2^15
    return torch.cat([p[0].to(dt) for p in parts]), torch.cat([p[1] for p in parts])


def _sampled(g, feature, label, per):
    """Sorted pixel indices with replacement: nine in ten on an object for depth maps,
    uniform for RGB images."""
    n = label.shape[0]
    out = []
    step = max(1, (1 << 24) // label[0].numel())
    for i in range(0, n, step):
        lb = label[i:i + step].reshape(-1, label[0].numel())
        if feature == "channel_diff":
            s = torch.randint(0, lb.shape[1], (lb.shape[0], per), generator=g, device=_DEV)
        else:
            obj = (lb > 1).float()
            p = obj * 0.9 / obj.sum(1, keepdim=True).clamp(min=1) + (1 - obj) * 0.1 / (1 - obj).sum(1, keepdim=True).clamp(min=1)
            s = torch.multinomial(p, per, replacement=True, generator=g)
        out.append(s.sort(1).values.to(torch.int32))
    return torch.cat(out)


def _np_image(feature, t):
    a = t.cpu().numpy()
    return a if feature == "channel_diff" else a.view(np.uint16)


def _sizes(case):
    """(count, width, height) of each group of same-size images of a case."""
    n, w, h = case["images"], case["width"], case["height"]
    if not (case.get("mixed") or case["what"] == "predict_batch"):
        return [(n, w, h)]
    third = n // 3
    return [(k, a, b) for k, a, b in ((n - 2 * third, w, h), (third, w // 2, h // 2), (third, w // 4, h // 4)) if k]


# -------------------------------------------------- features in plain torch ----
def _round_div(u, d):
    """round_half_away(u / d) for d > 0, exact in 64-bit floats."""
    q = (u.abs().double() / d.double() + 0.5).floor()
    return (q * u.sign()).to(torch.int64)


def _respond(feature, img, z, y, x, f):
    """Responses of features f[..., D] at pixels (z, y, x) of img [n][h][w]([3])."""
    n, h, w = img.shape[:3]
    if feature == "channel_diff":
        def read(dx, dy, c):
            xx, yy = x + dx, y + dy
            ok = (xx >= 0) & (xx < w) & (yy >= 0) & (yy < h)
            v = img.reshape(-1)[((z * h + yy.clamp(0, h - 1)) * w + xx.clamp(0, w - 1)) * 3 + c.clamp(0, 2)].to(torch.int64)
            return torch.where(ok, v, torch.zeros_like(v))

        return read(f[..., 2], f[..., 3], f[..., 0]) - read(f[..., 4], f[..., 5], f[..., 1])
    flat = img.reshape(-1)
    d = flat[(z * h + y) * w + x].to(torch.int64)
    d = torch.where(d == 0, torch.full_like(d, 10000), d)

    def probe(u, v):
        xx, yy = x + _round_div(u, d), y + _round_div(v, d)
        ok = (xx >= 0) & (xx < w) & (yy >= 0) & (yy < h)
        r = flat[(z * h + yy.clamp(0, h - 1)) * w + xx.clamp(0, w - 1)].to(torch.int64)
        return torch.where(ok & (r != 0), r, torch.full_like(r, 10000))

    return probe(f[..., 0], f[..., 1]) - probe(f[..., 2], f[..., 3])


def _forest(g, case):
    """Trees grown with one random feature and threshold per node on sampled pixels of a few
    images: (left children, features, thresholds, posteriors) of each, on the GPU."""
    feature, K, depth = case["feature"], case["classes"], case["depth"]
    b = _FEATURES[feature]
    D = len(b["low"])
    w, h = case["width"], case["height"]
    per = 2000
    count = max(4, min(100, 12 << max(0, depth - 8)))
    img, label = _images(g, feature, count, w, h, K)
    s = _sampled(g, feature, label, per).to(torch.int64)
    z = torch.arange(count, device=_DEV).repeat_interleave(per)
    s = s.reshape(-1)
    y, x = s // w, s % w
    cls = label.reshape(count, -1)[z, s].to(torch.int64) - 1
    lo, up = torch.tensor(b["low"], device=_DEV), torch.tensor(b["up"], device=_DEV)
    trees = []
    for _ in range(case["trees"]):
        nodes = (1 << depth) - 1
        lc = torch.full((nodes,), -2, dtype=torch.int64, device=_DEV)
        feat = (torch.rand(nodes, D, generator=g, device=_DEV, dtype=torch.float64) * (up - lo) + lo).floor().to(torch.int64)
        # thresholds near zero most of the time, as trained trees have them
        t = torch.rand(nodes, generator=g, device=_DEV, dtype=torch.float64) * 2 - 1
        thr = (t * t.abs() * b["thr"]).round().to(torch.int64)
        lc[0] = -1
        node = torch.zeros_like(z)
        counts = torch.zeros(nodes, K, dtype=torch.float64, device=_DEV)
        counts.index_put_((node, cls), torch.ones_like(cls, dtype=torch.float64), accumulate=True)
        alive = torch.ones_like(z, dtype=torch.bool)
        for level in range(1, depth):
            at = alive.nonzero().squeeze(1)
            if at.numel() == 0:
                break
            nd = node[at]
            right = (_respond(feature, img, z[at], y[at], x[at], feat[nd]) > thr[nd]).to(torch.int64)
            tot = torch.bincount(nd, minlength=nodes)
            rt = torch.bincount(nd, weights=right.double(), minlength=nodes).to(torch.int64)
            split = (rt > 0) & (rt < tot)
            ids = split.nonzero().squeeze(1)
            lc[ids] = 2 * ids + 1
            lc[2 * ids + 1] = -1
            lc[2 * ids + 2] = -1
            go = split[nd]
            node[at] = torch.where(go, 2 * nd + 1 + right, nd)
            counts.index_put_((node[at][go], cls[at][go]), torch.ones(int(go.sum()), dtype=torch.float64, device=_DEV),
                              accumulate=True)
            alive[at] = go
            alive &= torch.bincount(node[alive], minlength=nodes)[node] > 20
        post = (counts / counts.sum(1, keepdim=True).clamp(min=1)).to(torch.float32)
        trees.append((lc, feat, thr, post))
    return trees


def _predict_inputs(case, seed):
    """The forest and, per size, the images (and masks) of a prediction case."""
    g = _gen(seed)
    trees = _forest(g, case)
    groups = []
    for n, w, h in _sizes(case):
        img, label = _images(g, case["feature"], n, w, h, case["classes"])
        mask = (label > 1).to(torch.uint8) if case["mask"] else None
        groups.append((img, mask))
    return trees, groups


# --------------------------------------------------------------- the passes ----
def prepare(case, seed):
    what = case["what"]
    st = dict(case=case)
    if what == "train":
        g = _gen(seed)
        b = _FEATURES[case["feature"]]
        images = []
        for n, w, h in _sizes(case):
            img, label = _images(g, case["feature"], n, w, h, case["classes"])
            s = _sampled(g, case["feature"], label, case["samples"])
            px, lb, sm = _np_image(case["feature"], img), label.cpu().numpy(), s.cpu().numpy().view(np.uint32)
            images += [pg.TrainingSetImage(px[i], lb[i], case["classes"], sm[i]) for i in range(n)]
        st["config"] = pg.ForestConfig(case["feature"], case["classes"])
        st["params"] = pg.TreeTrainerParameters(case["features"], case["thresholds"], b["low"], b["up"], -b["thr"],
                                                b["thr"], case["min_leaf"])
        st["set"] = pg.TrainingSet(case["classes"], images)
        st["trainer"] = pg.TreeTrainer(st["config"])
        st["trainer"].upload(st["set"])
        st["id"] = int(seed) % 997
    elif what.startswith("predict"):
        trees, groups = _predict_inputs(case, seed)
        cfg = pg.ForestConfig(case["feature"], case["classes"])
        clf = pg.Classifier(cfg)
        for k, (lc, feat, thr, post) in enumerate(trees):
            t = pg.Tree(cfg, k, case["depth"])
            t.left_child[:] = lc.cpu().numpy()
            t.features[:] = feat.cpu().numpy()
            t.thresholds[:] = thr.cpu().numpy()
            t.posteriors[:] = post.cpu().numpy()
            clf << t
        st["classifier"] = clf
        if what == "predict_device":
            img, mask = groups[0]
            st["images"], st["mask"] = img, mask
            st["out"] = torch.zeros(case["images"], case["classes"], case["height"], case["width"], device=_DEV)
        else:
            st["images"] = [a for img, _ in groups for a in _np_image(case["feature"], img)]
            st["masks"] = [m for _, mask in groups for m in mask.cpu().numpy()] if case["mask"] else None
    elif what == "sample":
        g = _gen(seed)
        img, label = _images(g, "depth_diff2", case["images"], case["width"], case["height"], case["classes"])
        # a tenth of the pixels carry no label
        label[torch.rand(label.shape, generator=g, device=_DEV) < 0.1] = 0
        kind = pg.UniformImageSampler if case["kind"] == "uniform" else pg.ClassWeightedImageSampler
        args = () if case["kind"] == "uniform" else (case["classes"],)
        sampler = kind(case["samples"], *args, seed=int(seed) & 0xFFFF)
        st["sampler"] = sampler._c(2)
        st["context"] = pg.Classifier(pg.ForestConfig("depth_diff2", case["classes"]))
        st["images"], st["labels"] = img, label
        st["samples"] = torch.zeros(case["images"], sampler.stride, dtype=torch.int32, device=_DEV)
        st["counts"] = torch.zeros(case["images"], dtype=torch.int32, device=_DEV)
    else:
        g = _gen(seed)
        pal = _palette(case["classes"])
        n = case["images"] * case["width"] * case["height"]
        _, label = _depth_images(g, 1, case["width"], case["height"], case["classes"])
        table = torch.cat([torch.zeros(1, 3, dtype=torch.int64), torch.from_numpy(pal)]).to(_DEV)
        rgb = []
        for _ in range(case["images"]):  # each image: the label map shifted, one pixel in 50 of no class's colour
            lb = label[0].roll((int(torch.randint(0, case["height"], (1,), generator=g, device=_DEV)), 7), (0, 1))
            lb = torch.where(torch.rand(lb.shape, generator=g, device=_DEV) < 0.02, torch.zeros_like(lb), lb)
            c = table[lb.to(torch.int64)]
            rgb.append((c if case["channels"] == 3 else torch.cat([c, torch.full_like(c[..., :1], 255)], -1)).to(torch.uint8))
        st["rgb"] = torch.stack(rgb)
        st["map"] = np.ascontiguousarray(pal, np.uint8)
        st["context"] = pg.Classifier(pg.ForestConfig("depth_diff2", 2))
        st["out"] = torch.zeros(n, dtype=torch.uint8, device=_DEV)
    return st


def run(st):
    case = st["case"]
    what = case["what"]
    if what == "train":
        tree = pg.Tree(st["config"], st["id"], case["depth"])
        st["trainer"].train(tree, st["set"], st["params"])
        return dict(left_child=tree.left_child, features=tree.features, thresholds=tree.thresholds,
                    posteriors=tree.posteriors)
    if what == "predict":
        return st["classifier"].predict(st["images"][0], st["masks"][0] if st["masks"] else None)
    if what == "predict_batch":
        return st["classifier"].predict_batch(st["images"], st["masks"])
    if what == "predict_device":
        N.check(N.lib().pd_predict_posterior_device(
            st["classifier"].h, case["images"], st["images"].data_ptr(), case["width"], case["height"],
            None if st["mask"] is None else st["mask"].data_ptr(), st["out"].data_ptr()))
        return st["out"]
    if what == "sample":
        N.check(N.lib().pd_sample_device(
            st["context"].h, st["sampler"], case["images"], st["images"].data_ptr(), st["labels"].data_ptr(), case["width"],
            case["height"], st["samples"].shape[1], st["samples"].data_ptr(), st["counts"].data_ptr()))
        return dict(samples=st["samples"], counts=st["counts"])
    N.check(N.lib().pd_rgb_to_labels_device(st["context"].h, st["out"].numel(), st["rgb"].data_ptr(), case["channels"],
                                            st["map"].ctypes.data, case["classes"], st["out"].data_ptr(), None))
    return st["out"]


def work(case):
    what = case["what"]
    pixels = sum(n * w * h for n, w, h in _sizes(case))
    if what == "train":
        b = _FEATURES[case["feature"]]
        image = 3 if case["feature"] == "channel_diff" else 2
        samples = case["images"] * case["samples"]
        # every level down to the last splits most samples; one evaluation is two probes
        # (coordinates, bounds, address), their difference, a place among the thresholds and a count
        evals = samples * case["features"] * (case["depth"] - 1)
        node = 4 + (len(b["low"]) + 1) * 4 + case["classes"] * 4
        return dict(bytes=pixels * image + samples * 5 + ((1 << case["depth"]) - 1) * node, flops=evals * 20)
    if what.startswith("predict"):
        image = 3 if case["feature"] == "channel_diff" else 2
        return dict(bytes=pixels * (image + 4 * case["classes"] + (1 if case["mask"] else 0)),
                    flops=pixels * case["trees"] * (case["depth"] - 1) * 16)
    if what == "sample":
        return dict(bytes=pixels * 3 + case["images"] * case["samples"] * 4, flops=0)
    return dict(bytes=pixels * (case["channels"] + 1), flops=0)


def exact(case, seed):
    """Posteriors in 64 bits from the same forest and images; the other cases return whole
    numbers, or trees whose training takes too long here."""
    if not case["what"].startswith("predict"):
        return None
    trees, groups = _predict_inputs(case, seed)
    out = []
    for img, mask in groups:
        n, h, w = img.shape[:3]
        step = max(1, (1 << 22) // (h * w))
        for i in range(0, n, step):
            part = img[i:i + step]
            m = part.shape[0]
            q = torch.arange(m * h * w, device=_DEV)
            z, y, x = q // (h * w), q // w % h, q % w
            acc = torch.zeros(m * h * w, case["classes"], dtype=torch.float64, device=_DEV)
            for lc, feat, thr, post in trees:
                node = torch.zeros_like(q)
                for _ in range(1, case["depth"]):
                    c = lc[node]
                    right = (_respond(case["feature"], part, z, y, x, feat[node]) > thr[node]).to(torch.int64)
                    node = torch.where(c >= 0, c + right, node)
                acc += post[node].double()
            acc /= len(trees)
            if mask is not None:
                acc *= (mask[i:i + step].reshape(-1, 1) != 0)
            out += list(acc.view(m, h, w, -1).permute(0, 3, 1, 2))
    if case["what"] == "predict":
        return out[0]
    return out if case["what"] == "predict_batch" else torch.stack(out)
