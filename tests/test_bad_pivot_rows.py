"""Which row a covariance that is not positive definite is reported for: in each sub-block of a diagonal block, in
later blocks and in a ragged last one, in every precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def repeated(n, *rows):
    """Points far apart but for `rows`, which repeat point 0: with a noise of -s, s < v, K's pivots are close to v - s
    but for these rows', which are close to -2 s."""
    x = 10.0 * np.arange(n)
    x[list(rows)] = x[0]
    return x


FP64_ROWS = [(20, 1), (32, 31), (33, 32), (128, 40), (128, 75), (128, 100), (128, 127), (300, 128), (300, 190),
             (300, 255), (300, 256), (300, 290), (300, 299), (1000, 999)]


@pytest.mark.parametrize("n, row", FP64_ROWS)
def test_fp64(n, row):
    from gprat_b200 import capi

    rng = np.random.default_rng(n + row)
    y, h = rng.standard_normal(n), (1.0, 1.0, -0.1)
    gp = capi.CudaGP(repeated(n, row, *range(row + 1, n, 37)), y, 1, n, 1)
    for call in (lambda: gp.cholesky(h), lambda: gp.compute_loss(h),
                 lambda: gp.predict_with_uncertainty(h, rng.standard_normal(5), 1, 5)):
        with pytest.raises(capi.NotPositiveDefiniteError, match=rf"row {row}\)"):
            call()
    gp.cholesky((1.0, 1.0, 0.1))  # the handle stays usable


@pytest.mark.parametrize("n, row", [(128, 1), (128, 32), (128, 70), (128, 127), (384, 128), (384, 200), (384, 383)])
@pytest.mark.parametrize("precision", ["PREC_FP64_INT8", "PREC_MIXED_TF32", "PREC_MIXED_BF16"])
def test_tensor_core_modes(n, row, precision):
    from gprat_b200 import capi

    rng = np.random.default_rng(n + row)
    y, h, xt = rng.standard_normal(n), (1.0, 1.0, -0.1), rng.standard_normal(5)
    gp = capi.CudaGP(repeated(n, row, *range(row + 1, n, 37)), y, 1, n, 1)
    gp.set_precision(getattr(capi, precision))
    with pytest.raises(capi.NotPositiveDefiniteError, match=rf"row {row}\)"):
        gp.predict_with_uncertainty(h, xt, 1, 5)
    gp.predict_with_uncertainty((1.0, 1.0, 0.1), xt, 1, 5)
