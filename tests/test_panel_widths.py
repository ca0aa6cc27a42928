"""The factorisations with outer panels of several blocks: every way the recursion inside a panel can split, an odd
number of blocks, a ragged last block and a ragged last panel (the widths that large problems use, at small sizes)."""
import numpy as np
import pytest

from oracle import gprat_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [1, 2, 3, 4, 64])
@pytest.mark.parametrize("n, m", [(257, 30), (640, 65), (1030, 200), (1409, 7)])
def test_fp64(monkeypatch, n, m, blocks):
    from gprat_b200 import capi

    monkeypatch.setenv("GPRAT_CU_FP64_PANEL_BLOCKS", str(blocks))
    d = 6
    x, y, xt = O.synthetic(n, m, d)
    gp = capi.CudaGP(x, y, 1, n, d)
    for h in ((1.0, 1.0, 0.1), (1.5, 0.7, 0.2), (1.0, 1.0, 0.1)):  # eager, captured, replayed
        o = O.OracleGP(x, y, 1, n, d, h)
        om, ov = o.predict_with_uncertainty(xt, 1, m)
        mean, var = gp.predict_with_uncertainty(h, xt, 1, m)
        assert np.max(np.abs(mean - om)) <= 1e-10 * np.max(np.abs(om))
        assert np.max(np.abs(var - ov) / ov) <= 1e-10
    oloss, ograd = o.gradient()
    loss, grad = gp.loss_grad(h)  # with the rows of the identity along
    assert abs(loss - oloss) <= 1e-10 * abs(oloss)
    assert np.max(np.abs(grad - ograd)) <= 1e-10 * np.max(np.abs(ograd))
    assert abs(gp.compute_loss(h) - oloss) <= 1e-10 * abs(oloss)
    K = O.covariance(x, n, d, h)
    L = np.tril(gp.cholesky(h)[0].reshape(n, n))
    # |L L^T - K| <= (n + 1) eps |L||L^T|, |L||L^T| <= 1.1, and one ulp of K's exponentials
    assert np.max(np.abs(L @ L.T - K)) <= (n + 2) * np.finfo(float).eps * 1.1
    gp.close()


@pytest.mark.parametrize("blocks", [1, 2, 3, 4, 64])
@pytest.mark.parametrize("n, m", [(384, 30), (640, 300), (1408, 2100)])  # 3, 5 and 11 blocks of 128
def test_int8(monkeypatch, n, m, blocks):
    from gprat_b200 import capi

    monkeypatch.setenv("GPRAT_CU_OZ_PANEL_BLOCKS", str(blocks))
    d, h = 8, (1.0, 1.0, 0.1)
    x, y, xt = O.synthetic(n, m, d)
    om, ov = O.OracleGP(x, y, 1, n, d, h).predict_with_uncertainty(xt, 1, m)
    gp = capi.CudaGP(x, y, 1, n, d)
    gp.set_precision(capi.PREC_FP64_INT8)
    for _ in range(3):  # eager, captured, replayed
        mean, var = gp.predict_with_uncertainty(h, xt, 1, m)
        assert np.max(np.abs(mean - om)) <= 1e-8 * np.max(np.abs(om))  # the mode's stated error
        assert np.max(np.abs(var - ov) / ov) <= 1e-8
    gp.close()
