"""Gradients of needles (Gaussians hundreds of pixels long and half a pixel wide) do
not depend on the order in which the tiles add their sums.

The covariance's gradient is a difference of the conic's three sums that cancels by
the covariance's condition number (up to 10^6 here). Bar: two passes agree to 1e-4 of
the norm of the rotation's and the scales' gradients. The sums add a few thousand
partials in 64 bits (2^-53 * 4e3 * 10^6 < 1e-6); what is left is a last-place flip of
the covariance's gradient in 32 bits, which the rotation reads through components
smaller by the root of the condition number: 2^-24 * 10^3 = 6e-5.
"""
import numpy as np
import pytest

from rgsplat_b200 import api as R
from rgsplat_b200 import scenes

pytestmark = pytest.mark.gpu


def _passes(mode, views, count):
    rng = np.random.default_rng(5)
    g = scenes.random_gaussians(400, seed=3, mean_range=0.8)
    g[:, 3] = -1.0
    g[:, 8:11] = np.array([-0.3, -7.0, -7.0], np.float32)  # sigma 0.74 x 0.0009: 380 x 0.6 pixels
    cams = [scenes.look_at((0.3 - 0.4 * k, -0.2, -3.0), (0.0, 0.0, 0.0), 1280, 720, 1536.0) for k in range(views)]
    tr = R.Trainer(g, cams)
    for k in range(views):
        tr.set_target(k, rng.uniform(0.0, 1.0, (720, 1280, 4)).astype(np.float32))
    out = []
    for _ in range(count):
        tr.backward(list(range(views)), mode=mode)
        out.append(np.array(tr.grads(), np.float64).reshape(400, 60))
    tr.ctx.close()
    return out


@pytest.mark.parametrize("mode,views", [("PLAIN", 1), ("BATCHED", 3)])
def test_passes_agree(mode, views):
    out = _passes(getattr(R.Trainer, mode), views, 4)
    for k, name in ((slice(3, 7), "rotation"), (slice(7, 10), "log scale")):
        norm = np.linalg.norm(out[0][:, k])
        assert norm > 0
        worst = max(np.linalg.norm(o[:, k] - out[0][:, k]) for o in out[1:]) / norm
        assert worst < 1e-4, f"{name}: {worst:.2e}"
