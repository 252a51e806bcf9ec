"""z-scores of finite vectors whose standard deviation no bracket decides: far
outside the estimate's range, or on the midpoint of two floats."""
import numpy as np
import pytest

import tracetransform_gb300 as tt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-38, 1e-36, 1e-33, 1e-31, 1e30, 1e32, 1e35])
@pytest.mark.parametrize("n", [2, 33, 360])
def test_extreme_scales(oracle_lib, scale, n):
    x = (np.random.default_rng(n).standard_normal(n) * scale).astype(np.float32)
    want = oracle_lib.zscore(x)
    assert np.isfinite(want).all()
    assert np.array_equal(tt.zscore(x), want)


@pytest.mark.parametrize("e", [0, -20, 15])
def test_deviation_on_a_rounding_midpoint(oracle_lib, e):
    """a + b - (a + b) = 0 and a^2 + a b + b^2 = N^2 with N odd in (2^24, 2^25): the
    deviation of (a, b, -(a + b)) / 2 is N / 2, between two floats."""
    p, q = 3000, 2001
    a, b, big = p * p - q * q, 2 * p * q + q * q, p * p + p * q + q * q
    assert a * a + a * b + b * b == big * big and big % 2 and 2 ** 24 < big < 2 ** 25
    x = np.float32(2.0 ** (e - 1)) * np.array([a, b, -(a + b)], np.float32)
    assert x.astype(np.float64).sum() == 0
    assert (x.astype(np.float64) ** 2).sum() / 2 == (big * 2.0 ** (e - 1)) ** 2
    assert np.array_equal(tt.zscore(x), oracle_lib.zscore(x))
