"""The fixed-point reciprocal and power function of the primitive variables
against 50-digit decimals."""
import ctypes as C
from decimal import Decimal, getcontext

import numpy as np
import pytest

from magudi_gb300 import capi
from magudi_gb300.solver import load_library

pytestmark = pytest.mark.gpu

getcontext().prec = 50


def test_reciprocal_is_rounded_once():
    """Within 62 bits before its one rounding: 2^-53 (1 + 2^-8) of 1/x. Where
    1/x is not a normal number, and for zeros, infinities and NaN, the
    division's own result."""
    L = load_library()
    L.mgd_selftest_stencil.argtypes = [C.POINTER(C.c_double), C.c_int, C.c_int, C.c_int, C.POINTER(C.c_double)]
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(0.5, 2.0, 3000), 10.0 ** rng.uniform(-300, 300, 1000),
                        -(10.0 ** rng.uniform(-3, 3, 500)), 2.0 ** rng.integers(-1021, 1021, 200),
                        np.nextafter(1.0, [0.0, 2.0]), np.nextafter(2.0, [0.0, 3.0])])
    edge = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, 1.7e308, -1.7e308])
    w = np.zeros((x.size + edge.size, 9))
    w[:, 4] = np.concatenate([x, edge])
    out = np.zeros(len(w))
    assert L.mgd_selftest_stencil(capi.dptr(w), len(w), 0, 3, capi.dptr(out)) == 0
    for a, r in zip(x, out):
        assert abs(Decimal(float(r)) * Decimal(float(a)) - 1) <= Decimal(2) ** -53 * (1 + Decimal(2) ** -8), a
    with np.errstate(divide="ignore", over="ignore"):
        np.testing.assert_array_equal(out[x.size:], 1.0 / edge)


@pytest.mark.parametrize("n", [0.666, 0.76, 0.5, 1.0, 1.5, 1.999, 0.00390625])
def test_power_law_is_rounded_once(n):
    """Errors before the one rounding: log2 m to 2^-61 and the series' ends
    below 2^-59 in all, times n ln 2 < 1.4: 2^-53 (1 + 2^-5) of x^n inside
    [2^-400, 2^400); the FP64 form beyond it, below 2^-42 there (its
    logarithm carries one rounding of up to 700)."""
    L = load_library()
    L.mgd_selftest_pow.argtypes = [C.POINTER(C.c_double), C.c_int, C.c_double,
                                   C.POINTER(C.c_double), C.POINTER(C.c_double)]
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(0.5, 2.0, 600), 10.0 ** rng.uniform(-3, 3, 600), 2.0 ** rng.uniform(-399, 399, 300),
                        2.0 ** rng.integers(-390, 390, 60), np.nextafter(1.0, [0.0, 2.0]), [1.0],
                        2.0 ** np.array([-400.0, 399.99, -430.0, 430.0])])
    fast, ref = np.zeros_like(x), np.zeros_like(x)
    assert L.mgd_selftest_pow(capi.dptr(x), x.size, n, capi.dptr(fast), capi.dptr(ref)) == 0
    for a, f in zip(x, fast):
        exact = (Decimal(float(a)).ln() * Decimal(n)).exp()
        inside = 2.0 ** -400 <= a < 2.0 ** 400
        bound = Decimal(2) ** -53 * (1 + Decimal(2) ** -5) if inside else Decimal(2) ** -42
        assert abs(Decimal(float(f)) - exact) <= bound * exact, (a, f)


def test_power_law_outside_its_domain():
    """Zero, negative, infinite and undefined arguments as CUDA's pow."""
    L = load_library()
    x = np.array([0.0, -0.0, -1.5, np.inf, -np.inf, np.nan, 1e-310])
    fast, ref = np.zeros_like(x), np.zeros_like(x)
    assert L.mgd_selftest_pow(capi.dptr(x), x.size, 0.666, capi.dptr(fast), capi.dptr(ref)) == 0
    np.testing.assert_array_equal(fast, ref)
