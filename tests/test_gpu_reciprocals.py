"""The FP64 kernels' reciprocal and reciprocal square root (pg_hydro.cuh)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(-1e-30, 1e-30), (-4.0, 4.0), (-300.0, 300.0), (-1000.0, 1000.0)])
def test_inv_and_rsq_within_two_ulp(lo, hi):
    """Arguments 2^U(lo, hi), and those next to powers of two, where the last bit
    weighs most.  The iteration's own error is below 2^-57 (a start good to 2^-19,
    cubed); with the rounding of its last product and sum (half an ulp of the
    correction, half of the result, and that of y e in rsq) the result is within
    2 ulp = 2^-51 of the value."""
    from penguin_b200._lib import check, lib

    rng = np.random.default_rng(5)
    x = 2.0 ** rng.uniform(lo, hi, 200000)
    p = 2.0 ** np.floor(np.linspace(lo, hi, 1000))
    x = np.concatenate([x, p, np.nextafter(p, 0.0), np.nextafter(p, np.inf), 3.0 * p])
    out = np.empty(2 * x.size)
    dp = ctypes.POINTER(ctypes.c_double)
    check(lib().pg_test_inv_rsq(x.ctypes.data_as(dp), x.size, out.ctypes.data_as(dp)))
    xl = x.astype(np.longdouble)
    for got, want in ((out[0::2], 1 / xl), (out[1::2], 1 / np.sqrt(xl))):
        assert np.abs((got.astype(np.longdouble) - want) / want).max() <= 2.0**-51
