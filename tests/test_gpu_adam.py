"""The optimiser's branch-free quotients and root against the oracle's divisions,
over the whole range of moments: zeros, values on both sides of the limits between
the two forms (2^-100, 2^-60, 2^60), infinities and NaN, first and late steps, with
and without eps.

Bar: 4 ulp of the update (at most one each in the two bias corrections, the root
and the quotient). The parameters start at zero, so the update is read as it is;
the quaternion, which the step renormalises, is left to the other Adam tests."""
import numpy as np
import pytest

import oracle as O
from rgsplat_b200 import api as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-15, 1e-8, 0.0])
@pytest.mark.parametrize("t", [0, 1, 30_000])
@pytest.mark.parametrize("n", [1, 255, 4097])
def test_update_matches_oracle(n, t, eps):
    rng = np.random.default_rng(n + t)

    def wide(lo, hi, shape, signed=True):
        x = 10.0 ** rng.uniform(lo, hi, shape) * (rng.choice([-1.0, 1.0], shape) if signed else 1.0)
        x[rng.random(shape) < 0.2] = 0.0
        return x.astype(np.float32)

    # rows alternate between late training's range and every finite magnitude
    lo, hi = np.where(np.arange(n) % 2, -12.0, -36.0)[:, None], np.where(np.arange(n) % 2, -3.0, 18.0)[:, None]
    grads = wide(lo, hi, (n, 60))
    m1, m2 = wide(lo, hi, (n, 59)), wide(2 * lo.clip(-18), 2 * hi, (n, 59), signed=False)
    if n > 100:
        grads[7, 20], m1[9, 30], m2[11, 40], m2[13, 41], m1[15, 3] = np.nan, np.inf, np.inf, np.nan, -np.inf
    g0 = np.zeros((n, 59), np.float32)
    g0[:, 4] = 1.0
    out = {}
    for name, M in (("gpu", R), ("oracle", O)):
        g, st = g0.copy(), M.AdamState(n)
        st.m1[:], st.m2[:], st.t = m1.reshape(-1), m2.reshape(-1), t
        M.adam_step(g, grads, st, M.TrainConfig(eps=eps))
        out[name] = np.delete(g, range(4, 8), axis=1), st.m1.copy(), st.m2.copy()
    for a, b in zip(out["gpu"][1:], out["oracle"][1:]):
        assert np.array_equal(a, b, equal_nan=True)
    np.testing.assert_allclose(out["gpu"][0], out["oracle"][0], rtol=4 * 2.0**-23, atol=2.0**-126)
