"""Implied volatilities where the search leaves its usual range."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def R():
    import rbergomi_gb300 as R
    return R


def otm_call(K, T, s):
    """Out-of-the-money call by scaled complementary error functions: no cancellation, no underflow
    before the result's."""
    from scipy.special import erfcx
    v = s * math.sqrt(T)
    d1 = -math.log(K) / v + v / 2
    d2 = d1 - v
    return 0.5 * math.exp(-0.5 * d1 * d1) * (erfcx(-d1 / math.sqrt(2)) - erfcx(-d2 / math.sqrt(2)))


@pytest.mark.parametrize("K,T", [(1.2, 0.3), (2.0, 1.0), (8.0, 0.02)])
def test_prices_down_to_the_smallest_doubles(R, K, T):
    """d1 from -30 to -37 (prices 1e-199 to 1e-301): FP64 d1 leaves a few 2^-53 d1^2 of the
    price, a relative 2^-53 d1^2 / d1^2 of the volatility; 1e-13."""
    d = np.linspace(30.0, 37.0, 29)
    v = -d + np.sqrt(d * d + 2 * math.log(K))  # d1 = -d
    s = v / math.sqrt(T)
    p = np.array([otm_call(K, T, x) for x in s])
    assert p.min() < 1e-295
    iv = R.implied_vol(p, np.full(len(p), K), np.full(len(p), T))
    np.testing.assert_allclose(iv, s, rtol=1e-13)


def test_prices_below_the_normal_doubles(R):
    """Denormal prices: from 1e-318 on a few roundings of 2^-1075 are below 1e-5 of the
    price, and that over d1^2 = 1400 of the volatility."""
    from scipy.special import log_ndtr
    K, T = 3.0, 0.5
    s = np.linspace(0.0405, 0.0416, 45)
    v = s * math.sqrt(T)
    d1 = -math.log(K) / v + v / 2
    log_price = log_ndtr(d1) + np.log1p(-np.exp(math.log(K) + log_ndtr(d1 - v) - log_ndtr(d1)))
    ok = (log_price > math.log(1e-318)) & (log_price < math.log(1e-308))
    assert ok.sum() >= 10
    p = np.exp(log_price[ok])
    np.testing.assert_allclose(R.implied_vol(p, np.full(len(p), K), np.full(len(p), T)), s[ok], rtol=1e-8)


def test_no_volatility_for_strikes_and_maturities_that_are_no_numbers(R):
    nan, inf = np.nan, np.inf
    P, K, T = (a.ravel() for a in np.meshgrid([1e-300, 1e-10, 0.3, 0.9999], [nan, inf, 1.5], [nan, inf, 1.0], indexing="ij"))
    iv = R.implied_vol(P, K, T)
    ok = (K == 1.5) & (T == 1.0)
    assert np.all(np.isnan(iv[~ok]))
    assert np.all(np.isfinite(iv[ok]))


def test_at_the_money_with_a_vanishing_maturity(R):
    """No volatility of the search's range reaches a price above 1e-15 in 1e-300 years."""
    assert np.all(np.isnan(R.implied_vol([1e-15, 1e-10, 0.3, 0.9999], np.ones(4), np.full(4, 1e-300))))
