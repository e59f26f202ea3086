"""The FP64 walks' inverse square root on its own: the walks' tests compare whole forces to 1e-12 of the largest one
and would not see it lose several digits.

Its seed is short enough for an exact square and good to 2^-20, the iteration's own error is 5/16 of the cube of twice
that (2e-18), and what follows rounds once at full size (2^-53) and at 2^-19 of it: 1.13e-16 in all.  Roots are
checked in 80 bits, which adds 1e-19.
"""
import numpy as np
import pytest

from next_b200 import native

pytestmark = pytest.mark.gpu

BOUND = 1.15e-16


def relative_error(x, y):
    return float(np.max(np.abs(y.astype(np.longdouble) * np.sqrt(x.astype(np.longdouble)) - 1)))


def values(exponents, rng):
    """Random mantissas of each exponent, and the powers of two with their neighbours."""
    powers = np.exp2(exponents.astype(np.float64))
    near = [powers, np.nextafter(powers, 0), np.nextafter(powers, np.inf), np.nextafter(2 * powers, 0)]
    return np.concatenate([(powers * rng.uniform(1, 2, (64, powers.size))).ravel(), *near])


@pytest.mark.parametrize("lo,hi", [(-60, 60), (-958, -60), (60, 959)])
def test_inverse_root(lo, hi):
    x = values(np.arange(lo, hi + 1), np.random.default_rng(abs(lo)))
    assert relative_error(x, native.debug_inverse_root(x)) <= BOUND


def test_inverse_root_dense_mantissas():
    """Two octaves, every 2^-19 of them: all of the seed's intervals."""
    x = 1.0 + np.arange(3 << 19) / float(1 << 19)
    assert relative_error(x, native.debug_inverse_root(x)) <= BOUND


def test_inverse_root_past_the_ends():
    """Operands beyond the limits get the limit's exponent: zero, subnormal, infinite ones too."""
    tiny = np.array([0.0, 5e-324, 1e-310, 2.2250738585072014e-308, 2.0 ** -1000, 2.0 ** -961, np.nextafter(2.0 ** -960, 0)])
    huge = np.array([2.0 ** 961, 2.0 ** 1000, np.finfo(np.float64).max, np.inf])
    low, high = native.debug_inverse_root(tiny), native.debug_inverse_root(huge)
    assert np.all(low > 0.999999 * 2.0 ** 480) and np.all(low <= 2.0 ** 480)
    assert np.all(high > 0.999999 * 2.0 ** -480) and np.all(high <= 2.0 ** -480)
    edge = np.array([2.0 ** -960, 2.0 ** 960])
    np.testing.assert_array_equal(native.debug_inverse_root(edge), [2.0 ** 480, 2.0 ** -480])
