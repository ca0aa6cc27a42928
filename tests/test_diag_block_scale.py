"""The diagonal-block kernel on covariances far from 1: whatever it decides by the size of a block's entries is
decided from finished entries, and does not show in the factor."""
import numpy as np
import pytest

from oracle import gprat_oracle as O

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("scale", [0.95e-120, 1.5e-120, 4e-120])
@pytest.mark.parametrize("n", [64, 128, 300])
def test_diagonal_that_crosses_a_threshold_while_it_is_updated(n, scale):
    """K's diagonal entries, 1.1 scale, lie above 1e-120 and the pivots they end as (down to 0.1 scale) below it, or
    some of them: the same bits from run to run, and the factor of the unscaled matrix."""
    from gprat_b200 import capi

    d = 4
    x, y, _ = O.synthetic(n, 4, d)
    gp = capi.CudaGP(x, y, 1, n, d)
    h = (1.0, scale, 0.1 * scale)
    first = gp.cholesky(h)[0]
    for _ in range(20):
        assert np.array_equal(gp.cholesky(h)[0], first)
    L = np.tril(first.reshape(n, n)) / np.sqrt(scale)
    K = O.covariance(x, n, d, (1.0, 1.0, 0.1))
    # |L L^T - K| <= (n + 1) eps |L||L^T| entry by entry, |L||L^T| <= 1.1; two further ulps for K's own
    # exponentials and for the scale
    assert np.max(np.abs(L @ L.T - K)) <= (n + 3) * EPS * 1.1


def factor(n, scale, noise=0.125, l=4.0):
    from gprat_b200 import capi

    x, y, _ = O.synthetic(n, 4, 4)
    gp = capi.CudaGP(x, y, 1, n, 4)
    return np.tril(gp.cholesky((l, scale, noise * scale))[0].reshape(n, n))


@pytest.mark.parametrize("k", [-505, -400, -251, -250, -249, -200, -1, 200, 249, 250, 251, 400, 500])
@pytest.mark.parametrize("n", [33, 128, 300])
def test_a_power_of_four_scales_the_factor_exactly(n, k):
    """chol(4^k K) = 2^k chol(K) in every bit, as long as no entry becomes subnormal."""
    if n > 128 and k < -400:
        return  # the trailing matrix's small entries would be
    want = factor(n, 1.0)
    assert np.array_equal(factor(n, 4.0 ** k), want * 2.0 ** k)


@pytest.mark.parametrize("scale", [1e-298, 1e-305, 1e-308, 1e-310])
def test_subnormal_covariances_are_factored(scale):
    """K's entries and pivots down to 0.1 scale, of which the smallest are subnormal numbers."""
    n = 70
    L = factor(n, scale, l=1.0) / np.sqrt(scale)
    K = O.covariance(O.synthetic(n, 4, 4)[0], n, 4, (1.0, scale, 0.125 * scale))
    K = K * 2.0 ** 1000 / (scale * 2.0 ** 1000)
    # the factorisation's (n + 3) eps |L||L^T| and one unit of K's last place, here 2^-1074
    assert np.max(np.abs(L @ L.T - K)) <= (n + 3) * EPS * 1.125 + 2.0 ** -1000 / (scale * 2.0 ** 74)


@pytest.mark.parametrize("n", [64, 200])
def test_infinite_noise_leaves_the_prior(n):
    from gprat_b200 import capi

    x, y, xt = O.synthetic(n, 9, 4)
    gp = capi.CudaGP(x, y, 1, n, 4)
    mean, var = gp.predict_with_uncertainty((1.0, 1.5, np.inf), xt, 1, 9)
    assert np.all(mean == 0.0) and np.all(var == 1.5)
