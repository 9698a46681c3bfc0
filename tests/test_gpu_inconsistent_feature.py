"""Training with a user feature that is no function of its inputs: it answers the regrouping
of a level (a kernel without dynamic shared memory) otherwise than the histograms, so the
nodes of the next level hold other samples than the splits counted.  The call has to fail with
an error, before any kernel has indexed a table by a class count above its total, and the next
call has to work.  Every split kernel meets such nodes: small nodes of few and of many classes,
chunked nodes, and both again where thresholds are searched."""
import numpy as np
import pytest

import padenti_gb300 as pg

# the response is the pixel's value, its class; ANSWER is what the regrouping gets
SOURCE = r"""
__device__ feat_t computeFeature(const pd::ImageView &img, int2 c, const feat_t *f, unsigned featDim) {
  unsigned smem;
  asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(smem));
  int k = img.read(c.x, c.y, 0);
  const int top = CLASSES - 1;
  if (smem == 0u) k = ANSWER;
  return k * SCALE;
}
"""


def _train(K, answer, span, fuse_max):
    w, h = 16, 30
    rows = K * (h // K)  # the same number of rows, so of samples, for every class
    px = np.ascontiguousarray(np.broadcast_to((np.arange(h) % K)[:, None], (h, w)), np.uint16)
    ts = pg.TrainingSet(K, [pg.TrainingSetImage(px, (px + 1).astype(np.uint8), K, np.arange(rows * w, dtype=np.uint32))])
    src = SOURCE.replace("CLASSES", str(K)).replace("ANSWER", answer).replace("SCALE", str(span // K))
    tr = pg.TreeTrainer(pg.ForestConfig("user", K, source=src, shape="u16x1_i32x4"))
    tr.set_tuning("fuse_max", fuse_max)
    tree = pg.Tree(tr.config, 1, 4)
    tr.train(tree, ts, pg.TreeTrainerParameters(70, 24, [-9] * 4, [9] * 4, 0, span, 5))
    return tree


@pytest.mark.gpu
@pytest.mark.parametrize("answer", ["top - k", "0", "top", "k ^ 1", "(c.x & 1) ? k : top - k"])
@pytest.mark.parametrize("K,span,fuse_max", [(4, 1200, 65535), (4, 1200, 0), (4, 9000, 65535), (4, 9000, 0),
                                             (30, 1200, 65535), (30, 1200, 0), (30, 9000, 65535)])
def test_other_samples_than_counted(K, span, fuse_max, answer):
    with pytest.raises(pg.PadentiError, match="reassignment disagrees"):
        _train(K, answer, span, fuse_max)
    tree = _train(K, "k", span, fuse_max)  # the same feature, answering alike: a tree
    assert (tree.left_child >= 0).sum() == (3 if K == 4 else 7)
