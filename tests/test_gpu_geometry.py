"""The geometry pass over every size of a view group: the gradients of a batched
step are the sum of its views' own gradients, and the fused optimiser step moves
the Gaussians as the gradient pass and the separate optimiser do. One to nine
views: whole groups of four, one more, one less, one or two views alone.

Bars: each plane's gradients within 1e-5 of its 2-norm (float sums over at most a
few thousand pixel terms in another order; 64-bit sums of the views), the stepped
Gaussians within the trainer tests' bar for one step."""
import numpy as np
import pytest

from rgsplat_b200 import api as R
from tests.test_gpu_trainer import assert_steps_close, multi_view_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nviews", [1, 2, 3, 4, 5, 7, 8, 9])
def test_batched_gradients_are_the_sum_over_views(nviews):
    g, cams, targets = multi_view_scene(n=2500, seed=7)
    views = [v % len(cams) for v in range(nviews)]
    tr = R.Trainer(g, cams, targets)
    want = np.zeros((g.shape[0], 60))
    for v in views:
        tr.backward([v], mode=R.Trainer.PLAIN)
        want += tr.grads()
    losses = tr.backward(views, mode=R.Trainer.BATCHED)
    got = tr.grads()
    for a, b in ((0, 3), (3, 7), (7, 10), (10, 11), (11, 59), (59, 60)):
        assert np.linalg.norm(got[:, a:b] - want[:, a:b]) <= 1e-5 * np.linalg.norm(want[:, a:b]), (a, b)
    tr.apply_adam(R.TrainConfig(), denom_increment=nviews)
    fused = R.Trainer(g, cams, targets)
    assert np.allclose(fused.step(views, mode=R.Trainer.BATCHED), losses, rtol=1e-5, atol=1e-8)
    assert_steps_close(tr.gaussians(), fused.gaussians(), 1)
