"""The gradient's kernel at the number of regressors up to which a tile's series windows are staged in shared memory,
one above it, and far above."""
import numpy as np
import pytest

from oracle import gprat_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, d", [(130, 128), (130, 129), (65, 1), (300, 400)])
def test_gradient(n, d):
    from gprat_b200 import capi

    rng = np.random.default_rng(n + d)
    x, y, h = rng.standard_normal(n + d - 1), rng.standard_normal(n), (np.sqrt(d), 1.0, 0.1)
    loss, grad = capi.CudaGP(x, y, 1, n, d).loss_grad(h)
    oloss, ograd = O.OracleGP(x, y, 1, n, d, h).gradient()
    assert abs(loss - oloss) <= 1e-10 * abs(oloss)
    assert np.max(np.abs(grad - ograd)) <= 1e-10 * np.max(np.abs(ograd))
