"""Interior stencils in integer arithmetic against exact rational sums."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from magudi_gb300 import capi
from magudi_gb300.solver import load_library

pytestmark = pytest.mark.gpu

# coefficients of offsets 1..4 (first derivative) and 0..4 (composite dissipation)
D1 = {capi.SBP_48: ([672, -168, 32, -3], 840), capi.SBP_12: ([1, 0, 0, 0], 2),
      capi.SBP_24: ([8, -1, 0, 0], 12), capi.SBP_36: ([45, -9, 1, 0], 60)}
COMP = {capi.SBP_48: ([-70, 56, -28, 8, -1], 256), capi.SBP_12: ([-2, 1, 0, 0, 0], 2),
        capi.SBP_24: ([-6, 4, -1, 0, 0], 16), capi.SBP_36: ([-20, 15, -6, 1, 0], 64)}


def run(x, scheme, op):
    L = load_library()
    L.mgd_selftest_stencil.argtypes = [C.POINTER(C.c_double), C.c_int, C.c_int, C.c_int, C.POINTER(C.c_double)]
    out = np.zeros(len(x))
    assert L.mgd_selftest_stencil(capi.dptr(np.ascontiguousarray(x)), len(x), scheme, op, capi.dptr(out)) == 0
    return out


def coefficients(scheme, op):
    """(numerators of offsets -4..4, denominator)."""
    if op == 2:
        c, den = COMP[scheme]
        return [c[abs(j)] for j in range(-4, 5)], den
    c, den = D1[scheme]
    s = -1 if op else 1
    return [0 if j == 0 else s * (c[abs(j) - 1] if j > 0 else -c[abs(j) - 1]) for j in range(-4, 5)], den


def windows(kind, n, rng):
    if kind == "smooth":  # around the exponent boundary at 1
        return 1.0 + 1e-3 * np.sin(0.05 * np.arange(9)[None, :] + rng.uniform(0, 6, (n, 1)))
    if kind == "crossing":
        return np.sin(0.1 * (np.arange(9)[None, :] - rng.uniform(0, 8, (n, 1))))
    if kind == "nearly constant":
        return -2.5 - 1e-15 * rng.integers(0, 5, (n, 9))
    if kind == "mixed exponents":
        return np.ldexp(rng.uniform(-1, 1, (n, 9)), rng.integers(-70, 70, (n, 9)))
    if kind == "zeros and noise":
        return np.where(rng.random((n, 9)) < 0.4, 0.0, rng.uniform(-1, 1, (n, 9))) * np.where(
            rng.random((n, 9)) < 0.3, 1e-17, 1.0) * np.where(rng.random((n, 9)) < 0.5, -1.0, 1.0)
    e = {"small": -860, "below the integer range": -960, "subnormal": -1060, "large": 990}[kind]
    return np.ldexp(rng.uniform(-1, 1, (n, 9)), e + rng.integers(-8, 8, (n, 9)))


KINDS = ["smooth", "crossing", "nearly constant", "mixed exponents", "zeros and noise", "small",
         "below the integer range", "subnormal", "large"]


@pytest.mark.parametrize("scheme", [capi.SBP_48, capi.SBP_12, capi.SBP_24, capi.SBP_36])
@pytest.mark.parametrize("op", [0, 1, 2])
def test_interior_stencils_against_rational_sums(scheme, op):
    """Integer sums: each tap is off by less than one unit, 2^-61 of the power
    of two at or below the largest tap, so the sum by sum |c| / den of them
    (1750/840 at most), and the result is rounded once (half up, from 64 bits
    kept: 2^-53 (1 + 2^-8)). Outside that range the FP64 sum of nine products:
    below 16 roundings of the largest product, plus 16 subnormal units."""
    c, den = coefficients(scheme, op)
    total = Fraction(sum(abs(v) for v in c), den)
    for kind in KINDS:
        x = windows(kind, 257, np.random.default_rng(3))
        got = run(x, scheme, op)
        fp64 = kind in ("below the integer range", "subnormal")
        for w, g in zip(x, got):
            exact = sum(Fraction(v) * Fraction(float(t)) for v, t in zip(c, w)) / den
            top = Fraction(float(np.abs(w).max()))
            if fp64:
                bound = 16 * total * top / 2 ** 53 + 16 * Fraction(1, 2 ** 1074)
            else:
                bound = abs(exact) * (1 + Fraction(1, 256)) / 2 ** 53 + total * top / 2 ** 61
            assert abs(Fraction(float(g)) - exact) <= bound, (kind, w, g, float(exact))


@pytest.mark.parametrize("op", [0, 1, 2])
def test_fields_at_rest_and_non_finite_taps(op):
    x = np.zeros((4, 9))
    x[1] = -0.0
    x[2, 3], x[3, 7] = np.inf, np.nan
    got = run(x, capi.SBP_48, op)
    assert got[0] == 0.0 and got[1] == 0.0
    assert not np.isfinite(got[2]) and np.isnan(got[3])
    flat = run(np.full((3, 9), -0.3), capi.SBP_48, op)
    assert np.all(flat == 0.0)
