"""Pruned pair counts of fixed scenes of large splats. The counts are integers of the
scene: those that correctly rounded square roots and quotients give (approximate ones
move a pair or two in ten million in or out)."""
import numpy as np
import pytest

from rgsplat_b200 import api as R
from rgsplat_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,pairs", [(2, 13_308_115), (8, 13_543_065), (13, 13_784_110), (19, 14_477_929), (34, 15_429_005)])
def test_pairs(seed, pairs):
    n = 50_000
    g = scenes.random_gaussians(n, seed=seed, mean_range=1.5)
    g[:, 8:11] = np.random.default_rng(seed).uniform(-2.5, -0.5, (n, 3))
    w, h = 640 + seed, 480 + 2 * seed
    tr = R.Trainer(g.astype(np.float32), [scenes.look_at((0.3, 0.1, -3.0), (0.0, 0.0, 0.0), w, h, 1.1 * w)])
    tr.render(0)
    assert tr.ctx.stats()["pairs"] == pairs
    tr.ctx.close()
