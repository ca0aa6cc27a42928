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
