"""The quotient of the factor and per-step kernels (quot_nr) against 80-bit
division, over the operands that the kernels give it.

Tolerance: the reciprocal approximation is good to 2^-20 or better, so after one
Newton step to 2^-40, as is the quotient formed with it; its residual is exact
but for one rounding, so the correction leaves 2^-80 and the last addition's half
ulp.  The 80-bit quotient it is compared with is off by 2^-64 of itself, a 2^-11
of an ulp.  So 0.5 + 0.001 ulp; a product with the rounded reciprocal is off by
up to one and a half."""
import numpy as np
import pytest

from conftest import load_package

load_package()
from croma_fp_b200 import native  # noqa: E402

pytestmark = pytest.mark.gpu


def _worst(a, b):
    ref = a.astype(np.longdouble) / b.astype(np.longdouble)
    return float(np.max(np.abs(native.quot_check(a, b).astype(np.longdouble) - ref) / np.spacing(np.abs(ref).astype(np.float64))))


@pytest.mark.parametrize("operands", ["continuants", "faces", "photons"])
def test_quotient_within_half_an_ulp(operands):
    assert np.finfo(np.longdouble).nmant >= 63, "needs 80-bit floating point"
    rng = np.random.default_rng(11)
    n = 1 << 20
    mantissa = rng.uniform(1.0, 2.0, n)
    if operands == "continuants":      # theta_i-1 / theta_i: the pivot's inverse, both rescaled together
        a = mantissa * np.exp2(rng.integers(-40, 900, n))
        b = a * rng.uniform(1.0, 2.0, n) * np.exp2(rng.integers(0, 100, n))
    elif operands == "faces":          # |w| / (1 - exp(-|w|)), 1 / (exp(-|w| / 2) times the series)
        w = np.where(rng.random(n) < 0.5, rng.uniform(0.1, 1000.0, n), rng.uniform(0.0, 0.1, n))
        a = np.where(w < 0.1, 1.0, w)
        b = np.where(w < 0.1, np.exp(-0.5 * w) * (1.0 + w * w / 24.0 + w ** 4 / 1920.0), 1.0 - np.exp(-w))
    else:                              # e / (gamma - e), e^2 / (exp(X) - 1)
        a = 10.0 ** rng.uniform(-60.0, 6.0, n)
        b = 10.0 ** rng.uniform(-10.0, 90.0, n)
    assert _worst(a, b) <= 0.501


def test_quotient_of_nothing_and_of_powers_of_two():
    b = np.exp2(np.arange(-1000, 1001, dtype=np.float64))
    assert np.array_equal(native.quot_check(np.zeros_like(b), b), np.zeros_like(b))
    assert np.array_equal(native.quot_check(b, b), np.ones_like(b))
    assert native.quot_check(np.empty(0), np.empty(0)).size == 0
