"""The backward blend's accumulators against the oracle where its batches, its
groups and its decisions have their edges: image edges inside a tile, lists
around the 128-entry batch and the eight-splat group, opaque splats (alpha
clamped at 0.99, transmittance spent after a few), needles (ill-conditioned
conics, whose decisions the exact arithmetic takes), and a single splat.

The bar is the library's gradient tolerance, 1e-3 relative per accumulator:
an alpha is within 1e-6 relative of the forward's, and T is rebuilt through at
most a few hundred factors of 1 / (1 - alpha), each within 1e-6 / (1 - alpha)
<= 1e-4 (alpha <= 0.99) and on the average far below.
"""
import numpy as np
import pytest

import oracle as O
from rgsplat_b200 import api as R
from rgsplat_b200 import debug as D
from rgsplat_b200 import scenes

pytestmark = pytest.mark.gpu

TOL = 1e-3


def _scene(kind, n, w, h):
    g = scenes.random_gaussians(n, seed=n + w, mean_range=0.6)
    if kind == "opaque":
        g[:, 3] = np.random.default_rng(1).uniform(4.0, 9.0, n)
    elif kind == "needles":
        g[:, 8:11] = np.array([-6.5, -6.5, -0.5], np.float32)
    elif kind == "large":
        g[:, 8:11] = -1.0
        g[:, 3] = -3.0
    cam = scenes.look_at((0.3, -0.2, -3.0), (0.0, 0.0, 0.0), w, h, 1.2 * w)
    return g, cam


@pytest.mark.parametrize("tile,ppt", [((16, 16), 2), ((16, 16), 1), ((8, 32), 2), ((32, 8), 1)])
@pytest.mark.parametrize("kind,n,w,h", [("plain", 1, 16, 16), ("plain", 9, 17, 33), ("large", 127, 40, 23), ("large", 129, 31, 47),
                                        ("large", 600, 65, 16), ("opaque", 700, 70, 50), ("needles", 900, 64, 41)])
def test_accumulators_match_oracle(kind, n, w, h, tile, ppt):
    g, cam = _scene(kind, n, w, h)
    target = np.random.default_rng(7).uniform(0.0, 1.0, (h, w, 4)).astype(np.float32)
    ctx = R.Context(tile=tile, pixels_per_thread=ppt)
    acc, _ = D.backward(g, cam, target, (0.0, 0.0, 0.0), 0.2, ctx)
    ref = O.render_and_backward(g, cam, target, (0.0, 0.0, 0.0), 0.2)
    assert np.abs(ref.acc).max() > 0
    for k in range(9):
        want = np.asarray(ref.acc[:, k], np.float64)
        err = np.linalg.norm(acc[:, k] - want) / max(np.linalg.norm(want), 1e-30)
        assert err < TOL, f"accumulator {k}: {err:.2e}"
    ctx.close()
