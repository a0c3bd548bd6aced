"""The optimiser's step bit for bit against the oracle's divisions and root: moments,
gradients and parameters of every magnitude, subnormals and signed zeros among them,
first and late steps, with and without eps, a frozen group (rate 0)."""
import numpy as np
import pytest

import oracle as O
from rgsplat_b200 import api as R

pytestmark = pytest.mark.gpu


def _bits(x):
    x = np.ascontiguousarray(x, np.float32)
    return np.where(np.isnan(x), np.uint32(0x7FC00000), x.view(np.uint32))


@pytest.mark.parametrize("eps", [1e-15, 1e-8, 0.0])
@pytest.mark.parametrize("t", [0, 1, 500, 30_000])
@pytest.mark.parametrize("span", [(-12.0, -3.0), (-45.0, -28.0), (-38.0, 18.0)])
def test_bits(span, t, eps):
    n = 6000
    rng = np.random.default_rng(int(t + 10 * abs(span[0])))

    def wide(lo, hi, shape, signed=True):
        x = 10.0 ** rng.uniform(lo, hi, shape) * (rng.choice([-1.0, 1.0], shape) if signed else 1.0)
        x[rng.random(shape) < 0.15] = 0.0
        x = x.astype(np.float32)
        return np.where(rng.random(shape) < 0.5, np.copysign(x, np.float32(-1.0)), x) if signed else x

    grads = wide(*span, (n, 60))
    grads[::3] = 0.0  # unseen: their moments only decay
    m1, m2 = wide(*span, (n, 59)), wide(max(2 * span[0], -45.0), max(2 * span[1], -30.0), (n, 59), signed=False)
    m2[::31, ::7] *= np.float32(-1.0)  # a caller's own state: the root is NaN
    g0 = wide(*span, (n, 59))
    g0[:, 4:8] = rng.normal(size=(n, 4))
    out = []
    for M in (R, O):
        g, st = g0.copy(), M.AdamState(n)
        st.m1[:], st.m2[:], st.t = m1.reshape(-1), m2.reshape(-1), t
        M.adam_step(g, grads, st, M.TrainConfig(eps=eps, lr_opacity=0.0))
        out.append([_bits(g), _bits(st.m1), _bits(st.m2)])
    for a, b in zip(*out):
        assert np.array_equal(a, b), f"{np.count_nonzero(a != b)} of {a.size} differ"
