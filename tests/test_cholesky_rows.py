"""cholesky(): what a tile keeps alive, and the C entry points against each other."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def model(nt, t, d=8):
    from gprat_b200 import capi

    rng = np.random.default_rng(5)
    return capi.CudaGP(rng.standard_normal(nt * t + d - 1), rng.standard_normal(nt * t), nt, t, n_reg=d)


@pytest.mark.parametrize("nt, t, rows_apart", [(6, 50, False), (2, 2112, True), (9, 512, True)])
def test_a_tile_keeps_lower_tiles_alive_only(nt, t, rows_apart):
    gp = model(nt, t)
    tiles = gp.cholesky([1.0, 1.0, 0.1])
    for i in range(nt):
        for j in range(i + 1):
            owner = tiles[i * nt + j].base
            count = i + 1 if rows_apart else nt * (nt + 1) // 2
            assert owner.nbytes == count * t * t * 8 and owner.flags.owndata
    gp.close()


@pytest.mark.parametrize("nt, t", [(1, 1), (1, 77), (5, 40), (3, 300)])
def test_one_buffer_and_separate_rows_agree(nt, t):
    from gprat_b200 import capi

    gp = model(nt, t)
    h = np.array([1.0, 1.0, 0.1])
    dp = ctypes.POINTER(ctypes.c_double)
    out = np.full((nt, nt, t * t), np.nan)
    capi.check(capi.lib.gprat_cu_cholesky(gp._h, h.ctypes.data_as(dp), out.ctypes.data_as(dp)))
    tiles = gp.cholesky(h)
    for i in range(nt):
        for j in range(nt):
            if j <= i:
                assert np.array_equal(out[i, j], tiles[i * nt + j])
            else:
                assert tiles[i * nt + j] is None and np.all(out[i, j] == 0.0)
    with pytest.raises(capi.GpratCudaError):
        capi.check(capi.lib.gprat_cu_cholesky_rows(gp._h, h.ctypes.data_as(dp), (ctypes.c_void_p * nt)()))
    gp.close()
