"""The backward blend's alpha and its decision against 64 bits.

Alpha is the opacity times the special-function unit's exponential: its error is that
exponential's own plus one rounding of the product (2^-24) and the rounding of the
forward's exp that the exponential is measured against (2^-23), whatever the opacity.
The decision alpha >= 1/255 is taken without the forward's arithmetic only 4e-6 or
more from it (log2 units), half of which is kept for the forward's roundings.
"""
import pytest

from rgsplat_b200 import debug as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power_lo", [-0.25, -1.0, -5.5])
@pytest.mark.parametrize("opacity", [(1 / 254.9, 1 / 16), (1 / 16, 0.5), (0.5, 1.0)])
def test_alpha_error(power_lo, opacity):
    rel, decision = D.backward_alpha_error(power_lo, *opacity)
    assert rel <= D.exp_sfu_error(power_lo, 0.0, 1 << 22) + 2.0**-24 + 2.0**-23
    assert decision < 2e-6
