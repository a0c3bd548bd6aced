"""The blend kernels against the oracle where their batches, the backward's
groups and their decisions have their edges: image edges inside a tile, lists
around the 128-entry batch and the eight-splat group, opaque splats (alpha
clamped at 0.99, transmittance spent after a few), needles (ill-conditioned
conics, whose decisions the exact arithmetic takes), a single splat, a colour
that overflows to NaN, and as many tiles as pass from two to four pixels per
thread.

Images, final T and last contributors are the oracle's bit for bit. For the
backward's accumulators the bar is the library's gradient tolerance, 1e-3 relative per accumulator:
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
    elif kind == "overflow":
        g[:, 8:11] = -2.0
        g[::7, 11:59] = 3e38 * np.where(np.arange(48) % 2, 1.0, -1.0).astype(np.float32)
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


@pytest.mark.parametrize("tile,ppt", [((16, 16), 2), ((16, 16), 1), ((8, 32), 2), ((32, 8), 1)])
@pytest.mark.parametrize("kind,n,w,h", [("plain", 1, 16, 16), ("plain", 9, 17, 33), ("large", 129, 31, 47), ("large", 600, 65, 16),
                                        ("opaque", 700, 70, 50), ("needles", 900, 64, 41), ("overflow", 300, 48, 40),
                                        ("plain", 400, 1280, 800)])
def test_forward_is_the_oracles_bit_for_bit(kind, n, w, h, tile, ppt):
    g, cam = _scene(kind, n, w, h)
    ctx = R.Context(tile=tile, pixels_per_thread=ppt)
    for bg in ((0.0, 0.0, 0.0), (0.25, 0.5, 1.0)):
        rgb, final_t, last = D.forward(g, cam, bg, ctx)
        want = O.render_color(g, cam, bg)
        assert np.array_equal(rgb, want[0].reshape(rgb.shape), equal_nan=True)
        assert np.array_equal(final_t, want[1].reshape(final_t.shape))
        if tile == (16, 16):  # other tile shapes index their own lists
            assert np.array_equal(last, want[2].reshape(last.shape))
    ctx.close()
