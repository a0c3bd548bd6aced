"""Large host copies (several threads through page-locked slabs) return what the
small ones do: sizes on both sides of the 8 MiB threshold and of the 1 MiB chunk,
into fresh and used arrays, from several threads with a context each, and again
after the last context has given the slabs back. The slabs exist from the first
32 MiB of large copies on, which the first test brings about."""
import threading

import numpy as np
import pytest

from rgsplat_b200 import api as R
from rgsplat_b200 import scenes

pytestmark = pytest.mark.gpu

CAM = scenes.look_at((0.0, 0.0, -4.0), (0.0, 0.0, 0.0), 16, 16, 20.0)


def _round_trip(n, seed):
    g = np.random.default_rng(seed).normal(size=(n, 59)).astype(np.float32)
    tr = R.Trainer(g, [CAM])
    for _ in range(2):
        assert np.array_equal(tr.gaussians(), g)
    out = np.full((n, 59), 7.0, np.float32)
    got = R.C.c_size_t(0)
    tr.ctx.check(tr.lib.rgs_trainer_get_gaussians(tr.ctx.handle, R._fp(out), n, R.C.byref(got)))
    assert got.value == n and np.array_equal(out, g)
    tr.ctx.close()


def test_before_and_after_the_slabs_exist():
    for n in (35_545, 150_000, 35_545, 400_001):
        _round_trip(n, n)


@pytest.mark.parametrize("n", [35_544, 35_545, 39_988, 39_989, 100_003, 400_001])
def test_round_trip(n):
    big = R.Trainer(np.zeros((150_000, 59), np.float32), [CAM])  # 35 MB: the slabs exist
    _round_trip(n, n)
    big.ctx.close()


def test_threads_with_a_context_each():
    errors = []

    def run(k):
        try:
            for j in range(3):
                _round_trip(60_000 + 1000 * k, 10 * k + j)
        except BaseException as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(5)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_page_locked_arrays():
    torch = pytest.importorskip("torch")
    g = np.random.default_rng(1).normal(size=(50_000, 59)).astype(np.float32)
    pinned = torch.empty(50_000, 59, pin_memory=True)
    pinned.copy_(torch.from_numpy(g))
    tr = R.Trainer(pinned.numpy(), [CAM])
    assert np.array_equal(tr.gaussians(), g)
