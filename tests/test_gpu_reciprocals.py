"""The kernels' reciprocals and reciprocal square roots (pg_hydro.cuh, pg_f32.cuh)."""
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


@pytest.mark.parametrize("lo,hi", [(-4.0, 4.0), (-60.0, 60.0), (-100.0, -50.0), (50.0, 100.0)])
def test_root_of_a_product_in_fp32(lo, hi):
    """(a b)^-1/2 of factors 2^U(lo, hi), also where a b leaves the normal range: there two roots
    good to 2^-22.9 and the rounding of their product, else one root of a rounded product."""
    from penguin_b200._lib import check, lib

    rng = np.random.default_rng(6)
    ab = (2.0 ** rng.uniform(lo, hi, (200000, 2))).astype(np.float32)
    out = np.empty(len(ab), dtype=np.float32)
    fp = ctypes.POINTER(ctypes.c_float)
    check(lib().pg_test_root32(ab.ctypes.data_as(fp), len(ab), out.ctypes.data_as(fp)))
    want = 1.0 / np.sqrt(ab[:, 0].astype(np.float64) * ab[:, 1])
    assert np.abs(out / want - 1.0).max() <= 2.0 * 2.0**-22.9 + 2.0**-24
