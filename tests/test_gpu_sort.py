"""Tile lists' order at the sizes where the sort changes: one slot, the edges of a
warp, of a CTA's chunk in the cluster sort (8 CTAs, chunks of a multiple of 32), of
its largest size (65536) and past it, with one and with two digits of supertiles,
many equal depths (ties keep index order) and slots that are culled. The expected
lists are formed from the projection's depths and rectangles by numpy's stable
sort; lists are integers: equal."""
import numpy as np
import pytest

from rgsplat_b200 import api as R
from rgsplat_b200 import debug as D
from rgsplat_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(64, 48), (1700, 1300)])
@pytest.mark.parametrize("n", [1, 33, 255, 257, 8192, 8225, 40_001, 65_535, 65_536, 65_537])
def test_lists_are_in_depth_then_index_order(n, w, h):
    rng = np.random.default_rng(n)
    g = scenes.random_gaussians(n, seed=n, mean_range=1.0)
    g[:, 8:11] = -5.0  # a few pixels each
    g[:, 2] = rng.integers(-6, 7, n).astype(np.float32) / 4.0  # 13 depths, the front ones behind the camera
    cam = scenes.look_at((0.0, 0.0, -1.2), (0.0, 0.0, 0.0), w, h, 0.9 * w)
    ctx = R.Context()
    seen, rec, rect = D.project(g, cam, ctx)[:3]
    off, got = D.tile_lists(g, cam, ctx)
    order = np.flatnonzero(seen)
    order = order[np.argsort(rec[order, 9], kind="stable")]
    tw = (w + 15) // 16
    x0, y0, x1, y1 = (rect[order, k].astype(np.int64) for k in range(4))
    per = (x1 - x0) * (y1 - y0)
    splats = np.repeat(order, per)
    k = np.arange(per.sum()) - np.repeat(np.cumsum(per) - per, per)
    wide = np.repeat(np.maximum(x1 - x0, 1), per)
    tiles = (np.repeat(y0, per) + k // wide) * tw + np.repeat(x0, per) + k % wide
    by_tile = np.argsort(tiles, kind="stable")
    want_off = np.concatenate([[0], np.cumsum(np.bincount(tiles, minlength=off.size - 1))])
    assert np.array_equal(off, want_off)
    assert np.array_equal(got, splats[by_tile])
    ctx.close()
