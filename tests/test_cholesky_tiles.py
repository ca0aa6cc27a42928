"""The factor's tiles for several tilings of one matrix: a tile row that is
copied in one part or in several, one tile, odd tile sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_every_tiling_holds_the_same_factor():
    from gprat_b200 import capi

    n = 3000
    rng = np.random.default_rng(5)
    x, y = rng.standard_normal(n + 7), rng.standard_normal(n)
    factors = []
    for nt in (1, 3, 24, 40):  # tiles of 3000 (two parts of 64 MB), 1000, 125, 75
        t = n // nt
        gp = capi.CudaGP(x, y, nt, t, n_reg=8)
        tiles = gp.cholesky([1.0, 1.0, 0.1])
        gp.close()
        L = np.zeros((n, n))
        for i in range(nt):
            for j in range(nt):
                tile = tiles[i * nt + j]
                assert (tile is None) == (j > i)
                if j <= i:
                    assert tile.shape == (t * t,)
                    L[i * t:(i + 1) * t, j * t:(j + 1) * t] = tile.reshape(t, t)
        factors.append(np.tril(L))
    for L in factors[1:]:
        assert np.array_equal(L, factors[0])
