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


def test_entries_do_not_depend_on_the_rows_a_cta_takes():
    """With one tile the strict upper triangle holds K itself: matrices that are
    assembled 16 and 64 rows at a time agree where they share the series."""
    from gprat_b200 import capi

    rng = np.random.default_rng(6)
    x, y = rng.standard_normal(6160), rng.standard_normal(6160)
    upper = {}
    for n in (6144, 5120, 1027, 15):
        gp = capi.CudaGP(x[:n + 7], y[:n], 1, n, n_reg=8)
        upper[n] = np.triu(gp.cholesky([1.0, 1.0, 0.1])[0].reshape(n, n), 1)
        gp.close()
    for n in (5120, 1027, 15):
        assert np.array_equal(upper[n], upper[6144][:n, :n])
