"""The forward ends a tile once its pixels are opaque, also where rows of the tile lie
below the image: at 1064 rows the last tile row holds eight image rows, at 1056 none
does, so the view has 1/66 more tiles. Bar: half as much again (a tile row that walks
its whole lists costs as much again as the rest of an opaque view, or more)."""
import numpy as np
import pytest

from rgsplat_b200 import api as R
from rgsplat_b200 import scenes

pytestmark = pytest.mark.gpu


def _forward_ms(g, height):
    cam = scenes.look_at((0.0, 0.0, -5.0), (0.0, 0.0, 0.0), 1600, height, 2000.0)
    tr = R.Trainer(g, [cam], [np.full((height, 1600, 4), 0.5, np.float32)])
    times = []
    for k in range(18):
        tr.ctx.set_profiling(k >= 3)
        tr.backward([0], mode=R.Trainer.BATCHED)
        times.append(tr.ctx.stage_times(reset=True)["forward"])
    tr.ctx.close()
    return float(np.median(times[3:]))


def test_opaque_view_with_rows_below_the_image():
    g = scenes.random_gaussians(300_000, seed=1, mean_range=2.0)
    g[:, 3] = 8.0
    g[:, 8:11] = -2.0
    even, ragged = _forward_ms(g, 1056), _forward_ms(g, 1064)
    assert even > 0.0
    assert ragged < 1.5 * even, f"{ragged:.3f} ms against {even:.3f}"
