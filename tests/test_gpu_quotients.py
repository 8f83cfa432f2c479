"""The quotients by energy denominators against the divisions they stand in for."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _quotient(x, d, f32):
    from fermicc import _lib
    out = np.empty_like(x)
    dp = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
    assert _lib.load().fcc_test_quotient(dp(x), dp(d), x.size, f32, dp(out)) == 0
    return out


def _operands(n, lo, hi):
    """x over 10^lo..10^hi of either sign; d as orbital-energy differences are, and
    next to powers of two, where a reciprocal is hardest to round."""
    rng = np.random.default_rng(n)
    x = rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(lo, hi, n)
    d = -10.0 ** rng.uniform(-2, 2, n)
    near = np.nextafter(2.0 ** rng.integers(-6, 7, n // 4), 0.0) * (1 - rng.integers(0, 4, n // 4) * 2.0 ** -53)
    d[:n // 4] = -near
    return x, d


def test_fp64_quotient_is_the_division():
    x, d = _operands(1 << 22, -30, 2)
    assert np.array_equal(_quotient(x, d, 0), x / d)
    x[:5] = [0.0, -0.0, np.inf, -np.inf, np.nan]
    out = _quotient(x[:8], d[:8], 0)
    assert np.array_equal(out[:2], [0.0, 0.0]) and not np.isfinite(out[2:5]).any() and np.isfinite(out[5:]).all()


def test_fp32_quotient_is_the_division_to_a_rounding():
    # the quotient before the correction is within two last places and the
    # correction's error is 2^-23 of it: 2^-45 of the quotient beside one rounding
    x, d = (a.astype(np.float32).astype(np.float64) for a in _operands(1 << 22, -20, 2))
    out = _quotient(x, d, 1)
    assert np.all(np.abs(out - x / d) <= (2.0 ** -24 + 2.0 ** -44) * np.abs(x / d))
