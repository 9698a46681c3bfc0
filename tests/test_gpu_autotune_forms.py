"""The autotuner's cache tells the two forms of the histogram kernels apart (the threshold
range decides which runs), and leaves entries without a form or a version alone."""
import pytest

import padenti_gb300 as pg
from cases import depth_case


@pytest.mark.gpu
def test_entries_of_one_form_do_not_serve_the_other(tmp_path):
    cfg, ts, _, _ = depth_case(n_images=6, n_features=64, n_thresholds=10, parts=1)
    cache = tmp_path / "tune.txt"

    def tune(thr):
        tp = pg.TreeTrainerParameters(64, 10, [-60000] * 4, [60000] * 4, -thr, thr, 10)
        return pg.TreeTrainer(cfg).autotune(ts, tp, 6, cache=cache, max_trials=2)["from_cache"]

    assert [tune(500), tune(400), tune(3000), tune(500), tune(3000)] == [0, 1, 0, 1, 1]
    old = [line.replace("/rank/v2", "").replace("/search/v2", "") for line in cache.read_text().splitlines()]
    assert all("/v2" not in line for line in old)
    cache.write_text("\n".join(old) + "\n")
    assert tune(500) == 0
