"""Tile lists whose masks travel in the entries' sort keys against the form that
makes them after the sort (batches over 65536 supertiles), where either has its
edges: rectangles around the 15-column / 16-row limit of the packed spans and the
eight supertile rows a warp expands at a time, needles whose rectangle is mostly
empty, tile columns and rows that end inside a supertile, each tile shape, pruned
and not. Lists are integers: equal, and each pruned list an ordered subset of the
full one that leaves the image as it is (bit for bit)."""
import numpy as np
import pytest

import oracle as O
from rgsplat_b200 import api as R
from rgsplat_b200 import debug as D
from rgsplat_b200 import scenes

pytestmark = pytest.mark.gpu


def _scene(kind, n):
    g = scenes.random_gaussians(n, seed=n, mean_range=1.0)
    rng = np.random.default_rng(5)
    if kind == "limits":  # radii from one tile to the whole image
        g[:, 8:11] = rng.uniform(-4.0, 0.0, (n, 1)).astype(np.float32)
    elif kind == "needles":
        g[:, 8:11] = np.stack([rng.uniform(-1.0, 0.5, n), np.full(n, -5.5), np.full(n, -5.5)], 1)
    return g


@pytest.mark.parametrize("tile", [(16, 16), (8, 32), (32, 8)])
@pytest.mark.parametrize("kind,n,w,h", [("plain", 1, 16, 16), ("plain", 1500, 333, 190), ("limits", 513, 640, 1200),
                                        ("limits", 700, 1111, 77), ("needles", 1025, 517, 900)])
def test_masks_in_keys_and_masks_after_the_sort_agree(kind, n, w, h, tile):
    g = _scene(kind, n)
    cam = scenes.look_at((0.3, -0.2, -4.0), (0.0, 0.0, 0.0), w, h, 1.1 * w)
    ctx = R.Context(tile=tile)
    lists = {}
    for wide in (0, 1):
        ctx.check(ctx.lib.rgs_debug_wide_supertiles(ctx.handle, wide))
        for pruned in (False, True):
            lists[wide, pruned] = D.tile_lists(g, cam, ctx, pruned=pruned)
    for pruned in (False, True):
        for a, b in zip(lists[0, pruned], lists[1, pruned]):
            assert np.array_equal(a, b)
    (of, ef), (op, ep) = lists[0, False], lists[0, True]
    assert 0 < ep.size <= ef.size
    for t in range(of.size - 1):
        full = iter(ef[of[t]:of[t + 1]].tolist())
        assert all(x in full for x in ep[op[t]:op[t + 1]].tolist()), f"tile {t}"
    for wide in (0, 1):
        ctx.check(ctx.lib.rgs_debug_wide_supertiles(ctx.handle, wide))
        rgb = R.render_color(g, cam, (0.0, 0.0, 0.0), ctx=ctx)
        assert np.array_equal(rgb, O.render_color(g, cam)[0].reshape(rgb.shape))
    ctx.close()


def test_a_trainer_steps_alike_in_both_forms():
    g = _scene("limits", 800)
    cams = scenes.sphere_cameras(3, 4.0, [(320, 240), (200, 333)], 1.0)
    targets = [np.random.default_rng(i).uniform(0, 1, (c.height, c.width, 4)).astype(np.float32) for i, c in enumerate(cams)]
    losses = []
    for wide in (0, 1):
        tr = R.Trainer(g, cams, targets)
        tr.ctx.check(tr.lib.rgs_debug_wide_supertiles(tr.ctx.handle, wide))
        losses.append(tr.backward([0, 1, 2], mode=R.Trainer.BATCHED))
        st = tr.ctx.stats()
        assert 0 < st["visible"] <= st["supertile_entries"] <= st["pairs"]
    assert np.array_equal(losses[0], losses[1])
