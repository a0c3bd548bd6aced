"""The batch setting changes no kernel: it neither recaptures a step's graph nor is
timed again by the autotuner."""
import numpy as np
import pytest

from rgsplat_b200 import api as R
from rgsplat_b200 import scenes

pytestmark = pytest.mark.gpu


def test_batch_recaptures_nothing():
    cams = [scenes.look_at((0.2 * k, 0.0, -3.0), (0.0, 0.0, 0.0), 96, 64, 100.0) for k in range(2)]
    tr = R.Trainer(scenes.random_gaussians(500, seed=1, mean_range=0.7), cams, [np.full((64, 96, 4), 0.5, np.float32)] * 2)

    def captures():
        tr.backward([0, 1], mode=R.Trainer.BATCHED)
        return tr.ctx.stats()["graph_captures"]

    first = captures()
    for batch in (128, 512, 256):
        tr.ctx.set_tiling((16, 16), batch, 2)
        assert tr.ctx.options()["batch"] == batch
        assert captures() == first
    tr.ctx.set_tiling((16, 16), 256, 1)
    assert captures() == first + 1
    pick, table = tr.autotune([0, 1], reps=1)
    assert tr.ctx.stats()["graph_captures"] - (first + 1) <= 6
    for tile in ("16x16", "8x32", "32x8"):
        for ppt in (1, 2):
            assert len({e["ms"] for e in table if (e["tile"], e["pixels_per_thread"]) == (tile, ppt)}) == 1
    tr.ctx.close()
