"""The FP64 update and panel solve at the edges of their tiles, boxes and chunks, and the factorisation that runs
both with a second row group and a vector along, at the edges of its panels."""
import numpy as np
import pytest

from oracle import gprat_oracle as O

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("tile", [0, 1, 2])
@pytest.mark.parametrize("m0, m1, N, K, lower", [
    (1, 0, 1, 1, True), (33, 0, 33, 7, True), (65, 40, 64, 8, True), (128, 1, 128, 16, True),
    (200, 31, 70, 24, True), (257, 130, 257, 129, True), (0, 65, 63, 130, False), (64, 64, 64, 512, False),
    (31, 97, 129, 50, False),
])
def test_update(tile, m0, m1, N, K, lower):
    from gprat_b200 import capi

    rng = np.random.default_rng(m0 + 7 * N + K)
    A0, A1, B, C0, C1 = (rng.standard_normal(s) for s in ((m0, K), (m1, K), (N, K), (m0, N), (m1, N)))
    z, y = rng.standard_normal(K), rng.standard_normal(N)
    g0, g1, gy = C0.copy(), C1.copy(), y.copy()
    capi.test_dgemm_update(A0, A1, B, g0, g1, lower, z, gy, tile)
    keep = np.tril(np.ones((m0, N), bool)) if lower else np.ones((m0, N), bool)
    # K products and sums in any order: an entry is off by at most (K + 1) eps of the sum of magnitudes
    bound = (K + 1) * EPS
    assert np.all(np.abs(g0 - (C0 - A0 @ B.T))[keep] <= (bound * (np.abs(C0) + np.abs(A0) @ np.abs(B).T))[keep])
    assert np.array_equal(g0[~keep], C0[~keep])
    assert np.all(np.abs(g1 - (C1 - A1 @ B.T)) <= bound * (np.abs(C1) + np.abs(A1) @ np.abs(B).T))
    assert np.all(np.abs(gy - (y - B @ z)) <= bound * (np.abs(y) + np.abs(B) @ np.abs(z)))


@pytest.mark.parametrize("tile", [0, 1, 2, 4])
@pytest.mark.parametrize("m0, m1, bs", [(1, 0, 1), (15, 17, 15), (16, 64, 16), (65, 33, 17), (128, 1, 127),
                                        (100, 129, 128), (0, 70, 50), (0, 0, 128)])
def test_solve(tile, m0, m1, bs):
    from gprat_b200 import capi

    rng = np.random.default_rng(m0 + 3 * m1 + bs)
    P0, P1 = rng.standard_normal((m0, bs)), rng.standard_normal((m1, bs))
    Linv = np.tril(rng.standard_normal((bs, bs)))
    rowsq, y = rng.uniform(1.0, 2.0, max(m1, 1)), rng.standard_normal(bs)
    g0, g1, gr, gy = P0.copy(), P1.copy(), rowsq.copy(), y.copy()
    capi.test_dgemm_solve(g0, g1, Linv, gr, gy, tile)
    bound = (bs + 1) * EPS
    for got, P in ((g0, P0), (g1, P1)):
        assert np.all(np.abs(got - P @ Linv.T) <= bound * (np.abs(P) @ np.abs(Linv).T))
    # the squares of the values it stored, summed in any order
    want = rowsq[:m1] + (g1 * g1).sum(axis=1)
    assert np.all(np.abs(gr[:m1] - want) <= (bs + 2) * EPS * want)
    assert np.all(np.abs(gy - Linv @ y) <= bound * (np.abs(Linv) @ np.abs(y)))


@pytest.mark.parametrize("n, m", [(128, 1), (129, 63), (256, 65), (257, 30), (511, 129), (640, 16), (1030, 200)])
def test_factorisation_with_rows_along(n, m):
    from gprat_b200 import capi

    d, h = 6, (1.0, 1.0, 0.1)
    x, y, xt = O.synthetic(n, m, d)
    o = O.OracleGP(x, y, 1, n, d, h)
    om, ov = o.predict_with_uncertainty(xt, 1, m)
    oloss, ograd = o.gradient()
    gp = capi.CudaGP(x, y, 1, n, d)
    for _ in range(3):  # eager, then captured and replayed
        mean, var = gp.predict_with_uncertainty(h, xt, 1, m)
        assert np.max(np.abs(mean - om)) <= 1e-10 * np.max(np.abs(om))
        assert np.max(np.abs(var - ov) / ov) <= 1e-10
    assert np.max(np.abs(gp.predict(h, xt, 1, m) - om)) <= 1e-10 * np.max(np.abs(om))
    assert abs(gp.compute_loss(h) - oloss) <= 1e-10 * abs(oloss)
    loss, grad = gp.loss_grad(h)
    assert abs(loss - oloss) <= 1e-10 * abs(oloss)
    assert np.max(np.abs(grad - ograd)) <= 1e-10 * np.max(np.abs(ograd))
