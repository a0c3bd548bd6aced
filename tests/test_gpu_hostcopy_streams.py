"""Large host copies on cudaStreamPerThread (handle 2), which is another stream in
every thread: they stay behind the calling thread's kernels."""
import numpy as np
import pytest

from rgsplat_b200 import api as R
from rgsplat_b200 import scenes

pytestmark = pytest.mark.gpu


def test_per_thread_stream():
    g = np.random.default_rng(2).normal(size=(150_000, 59)).astype(np.float32)
    cam = scenes.look_at((0.0, 0.0, -4.0), (0.0, 0.0, 0.0), 64, 64, 80.0)
    tr = R.Trainer(g, [cam], [np.full((64, 64, 4), 0.5, np.float32)])
    tr.ctx.set_stream(2)
    for k in range(4):
        tr.step([0])
        first = tr.gaussians()
        assert np.array_equal(tr.gaussians(), first)
        back = g + np.float32(k)
        tr.set_gaussians(back)
        assert np.array_equal(tr.gaussians(), back)
    tr.ctx.set_stream(None)
    tr.ctx.close()
