"""The reciprocal of the primitive variables is the division's, bit by bit."""
import ctypes as C

import numpy as np
import pytest

from magudi_gb300 import capi
from magudi_gb300.solver import load_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["significands", "exponents", "near ties"])
def test_reciprocal_is_bitwise_the_division(kind):
    L = load_library()
    L.mgd_selftest_stencil.argtypes = [C.POINTER(C.c_double), C.c_int, C.c_int, C.c_int, C.POINTER(C.c_double)]
    rng = np.random.default_rng(17)
    if kind == "significands":
        x = rng.uniform(0.5, 2.0, 400000)
        x[:4] = 1.0, np.nextafter(1.0, 0.0), np.nextafter(1.0, 2.0), np.nextafter(2.0, 0.0)
    elif kind == "exponents":
        x = np.ldexp(rng.uniform(0.5, 1.0, 200000), rng.integers(-1030, 1025, 200000)) * rng.choice([-1.0, 1.0], 200000)
    else:
        # 1/x halfway between two doubles to 2^-53 of their distance: x (Q + 1/2) near 2^105 in units of x's last bit
        q = rng.integers(2 ** 52, 2 ** 53, 100000)
        x = np.array([float(2 ** 106 // (2 * int(v) + 1) + k) for v, k in zip(q, rng.integers(-1, 2, len(q)))])
        x = np.ldexp(x, -52)
    w = np.zeros((x.size, 9))
    w[:, 4] = x
    out = np.zeros(x.size)
    assert L.mgd_selftest_stencil(capi.dptr(w), len(w), 0, 3, capi.dptr(out)) == 0
    with np.errstate(over="ignore", divide="ignore"):
        assert np.array_equal(out.view(np.int64), (1.0 / x).view(np.int64))
