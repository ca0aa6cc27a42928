"""The 128 x 128 diagonal-block kernel (factor and inverse) at the edges of its
32-wide sub-blocks, alone (n <= 128) and as the last, ragged block."""
import numpy as np
import pytest

from oracle import gprat_oracle as O

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 96, 97, 127, 128, 129, 161, 255])
def test_factor_and_inverse(n):
    from gprat_b200 import capi

    m, d, h = 40, 4, (1.0, 1.5, 0.05)
    x, y, xt = O.synthetic(n, m, d)
    gp = capi.CudaGP(x, y, 1, n, d)
    tile = gp.cholesky(h)[0].reshape(n, n)
    K = O.covariance(x, n, d, h)
    L = np.tril(tile)
    # a backward-stable factorisation: |L L^T - K| <= (n + 1) eps |L||L^T| entry by entry, and
    # |L||L^T| <= the largest diagonal entry of K; one further ulp of K for its own exponentials
    bound = (n + 2) * EPS * (h[1] + h[2])
    assert np.max(np.abs(L @ L.T - K)) <= bound
    # the strict upper triangle keeps K
    assert np.max(np.abs(np.triu(tile, 1) - np.triu(K, 1)), initial=0.0) <= 4 * EPS * h[1]
    # the inverse, through the solves that use it
    o = O.OracleGP(x, y, 1, n, d, h)
    om, ov = o.predict_with_uncertainty(xt, 1, m)
    mean, var = gp.predict_with_uncertainty(h, xt, 1, m)
    cond = (n * h[1] + h[2]) / h[2]  # bounds K's condition number
    assert np.max(np.abs(mean - om)) <= 8 * n * EPS * cond * np.max(np.abs(y))
    assert np.max(np.abs(var - ov)) <= 8 * n * EPS * cond * h[1]


@pytest.mark.parametrize("n, noise, row", [(40, -1.6, 1), (128, -1.6, 1), (200, -1.6, 1)])
def test_first_bad_pivot_is_reported(n, noise, row):
    from gprat_b200 import capi

    x, y, _ = O.synthetic(n, 4, 4)
    gp = capi.CudaGP(x, y, 1, n, 4)
    with pytest.raises(capi.NotPositiveDefiniteError, match=f"row {row - 1}"):
        gp.cholesky((1.0, 1.5, noise))
    gp.cholesky((1.0, 1.5, 0.05))  # the handle stays usable


@pytest.mark.parametrize("scale", [1e-280, 1e-295, 1e280, 1e295])
def test_pivots_at_the_ends_of_the_range(scale):
    """Pivots whose approximate reciprocal would be subnormal or infinite."""
    from gprat_b200 import capi

    n, d = 70, 4
    x, y, _ = O.synthetic(n, 4, d)
    gp = capi.CudaGP(x, y, 1, n, d)
    L1 = np.tril(gp.cholesky((1.0, 1.0, 0.125))[0].reshape(n, n))
    Ls = np.tril(gp.cholesky((1.0, scale, 0.125 * scale))[0].reshape(n, n))
    # sqrt(scale) L, to the rounding of the factorisation (cond(K) <= (n + 1/8) * 8)
    assert np.max(np.abs(Ls / np.sqrt(scale) - L1)) <= 8 * n * n * EPS * 8
