"""The reciprocals of the diagonal block's pivots over the range they are used in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_reciprocals_against_division():
    from gprat_b200 import capi

    rng = np.random.default_rng(1)
    exps = np.repeat(np.arange(-1022, 503), 64)
    mant = rng.uniform(1.0, 2.0, exps.size)
    mant[0::16] = 1.0
    mant[1::16] = np.nextafter(1.0, 2.0)
    mant[2::16] = np.nextafter(2.0, 1.0)
    mant[3::16] = 1.0 + 2.0 ** -20 * rng.integers(1, 2 ** 20, mant[3::16].size)  # the approximation sees no more bits
    d = np.ldexp(mant, exps)
    seed, inv, quotient = capi.test_pivot_reciprocals(d)
    exact = 1.0 / d
    assert np.array_equal(quotient, exact)
    e = 1 - np.longdouble(d) * np.longdouble(seed)  # 64 bits: good to 2^-62
    print("largest error of the approximation: 2^%.2f" % np.log2(float(np.max(np.abs(e)))))
    assert np.max(np.abs(e)) <= 2.0 ** -19
    # e^3 <= 2^-57 of the result is cut off and y + y (e + e^2) is rounded once (e + e^2's own roundings are
    # 2^-72): within 0.5 + 2^-4 ulp of 1 / d, so at most one ulp from the quotient
    ulps = np.abs(inv - exact) / np.spacing(exact)
    print("differs from the quotient in %d of %d, by at most %g ulp" % (np.count_nonzero(ulps), d.size, ulps.max()))
    assert ulps.max() <= 1.0
