"""Interior stencils in integer arithmetic: the forms that take several fields
or axes at once, and taps of very different size."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from magudi_gb300 import capi
from magudi_gb300.solver import load_library
from test_gpu_stencil import KINDS, coefficients, run, windows

pytestmark = pytest.mark.gpu

SCHEMES = [capi.SBP_48, capi.SBP_12, capi.SBP_24, capi.SBP_36]
FIELDS = {0: 3, 1: 4, 4: 1}


def run_groups(x, n, scheme, form):
    L = load_library()
    L.mgd_selftest_stencil_group.argtypes = [C.POINTER(C.c_double), C.c_int, C.c_int, C.c_int, C.POINTER(C.c_double)]
    out = np.zeros(n * FIELDS.get(form, 1))
    assert L.mgd_selftest_stencil_group(capi.dptr(np.ascontiguousarray(x)), n, scheme, form, capi.dptr(out)) == 0
    return out


def rational(c, den, w):
    return sum(Fraction(v) * Fraction(float(t)) for v, t in zip(c, w)) / den


def boxes(axes):
    """Boxes of 9 points along every axis (x fastest) whose axes through the
    centre hold the given windows (n, nD, 9); the other points are NaN."""
    n, nD, _ = axes.shape
    box = np.full((n,) + (9,) * nD, np.nan)
    for d in range(nD):
        line = [slice(None)] + [4] * nD
        line[nD - d] = slice(None)
        box[tuple(line)] = axes[:, d]
    return box.reshape(n, -1)


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("form", [0, 1, 4])
def test_fields_together_are_bitwise_the_fields_alone(scheme, form):
    """A field's sum does not depend on the other fields': beside ordinary ones
    some leave the integers' range, are at rest or cancel. And the persistent
    batch, which takes one field at a time, forms the same sums."""
    K = FIELDS[form]
    rng = np.random.default_rng(11)
    kinds = KINDS + ["rest", "cancel"]
    x = np.zeros((300, K, 9))
    for g in range(len(x)):
        for k in range(K):
            kind = kinds[rng.integers(len(kinds))]
            if kind == "cancel":
                x[g, k] = np.ldexp(rng.uniform(-1, 1, 9), -40)
                x[g, k, [2, 6]] = rng.uniform(1, 2)
            elif kind != "rest":
                x[g, k] = windows(kind, 1, rng)[0]
    alone = run(x.reshape(-1, 9), scheme, form % 4)
    together = run_groups(x, len(x), scheme, form)
    assert np.array_equal(together.view(np.int64), alone.view(np.int64))


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("nD", [2, 3])
def test_dissipation_over_the_axes_against_rational_sums(scheme, nD):
    """Each tap off by less than one unit, 2^-61 of the largest tap, and one
    rounding (half up, from 64 bits kept); below the integers' range 16
    roundings of the products of nine taps per axis and 16 subnormal units."""
    c, den = coefficients(scheme, 2)
    total = nD * Fraction(sum(abs(v) for v in c), den)
    real = [j for j in range(9) if c[j]]
    for kind in KINDS:
        axes = windows(kind, 101 * nD, np.random.default_rng(5)).reshape(101, nD, 9).copy()
        axes[:, :, 4] = axes[:, :1, 4]
        got = run_groups(boxes(axes), len(axes), scheme, nD)
        for w, g in zip(axes, got):
            exact = sum(rational(c, den, a) for a in w)
            top = Fraction(float(np.abs(w[:, real]).max()))
            if kind in ("below the integer range", "subnormal"):
                bound = 16 * nD * total * top / 2 ** 53 + 16 * Fraction(1, 2 ** 1074)
            else:
                bound = abs(exact) * (1 + Fraction(1, 256)) / 2 ** 53 + total * top / 2 ** 61
            assert abs(Fraction(float(g)) - exact) <= bound, (kind, w, g, float(exact))


@pytest.mark.parametrize("scheme", SCHEMES[1:])
@pytest.mark.parametrize("op", [0, 1, 2])
def test_taps_outside_a_narrow_stencil_do_not_set_its_unit(scheme, op):
    """The lower-order schemes' stencils are stored in the widest one's shape.
    Taps that their coefficients leave out may be 2^20 to 2^80 times the
    others: the sum is as exact as without them."""
    c, den = coefficients(scheme, op)
    total = Fraction(sum(abs(v) for v in c), den)
    real = np.array([v != 0 for v in c]) | (np.arange(9) == 4)
    rng = np.random.default_rng(7)
    x = rng.uniform(-1, 1, (400, 9))
    x[:, ~real] *= 2.0 ** rng.uniform(20, 80, (400, 1))
    x[200:, real] *= np.where(rng.random((200, int(real.sum()))) < 0.5, 0.0, -1.0)
    for w, g in zip(x, run(x, scheme, op)):
        exact = rational(c, den, w)
        top = Fraction(float(np.abs(w[real]).max()))
        bound = abs(exact) * (1 + Fraction(1, 256)) / 2 ** 53 + total * top / 2 ** 61
        assert abs(Fraction(float(g)) - exact) <= bound, (w, g, float(exact))
    # an undefined tap shows in the result, stencil or padding
    x = np.ones((9, 9))
    x[np.arange(9), np.arange(9)] = np.nan
    x = np.delete(x, 4, axis=0)
    assert np.all(np.isnan(run(x, scheme, op)))


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("op", [0, 1, 2])
def test_large_opposite_taps_that_cancel(scheme, op):
    """Large opposite taps whose difference (first derivatives) or sum
    (dissipation) is exactly zero leave what the small ones give. Bound: that
    of the FP64 sum over pairs, at most 16 roundings of the pairs' products."""
    c, den = coefficients(scheme, op)
    rng = np.random.default_rng(9)
    n = 400
    x = rng.uniform(-1, 1, (n, 9)) * 2.0 ** -rng.uniform(12, 90, (n, 1))
    for k in range(n):
        big = [j for j in range(1, 5) if rng.random() < 0.5] or [1]
        for j in big:
            v = rng.uniform(0.5, 2.0) * rng.choice([-1.0, 1.0])
            x[k, 4 + j], x[k, 4 - j] = v, (-v if op == 2 else v)
    x[::7, 4] = 0.0
    for w, g in zip(x, run(x, scheme, op)):
        exact = rational(c, den, w)
        f = [Fraction(float(t)) for t in w]
        pairs = sum(abs(c[4 + j]) * abs(f[4 + j] - f[4 - j] if op < 2 else f[4 + j] + f[4 - j]) for j in range(1, 5))
        pairs = (pairs + abs(c[4]) * abs(f[4])) / den
        assert abs(Fraction(float(g)) - exact) <= 16 * pairs / 2 ** 53, (w, g, float(exact))


@pytest.mark.parametrize("scheme", SCHEMES)
def test_mirrored_fields(scheme):
    """About a point a field is even about, its derivative is 0; about a point
    it is odd about, its dissipation is 0, along one axis and over several;
    zeros of either sign beside them change nothing."""
    rng = np.random.default_rng(13)
    h = rng.uniform(-1, 1, (200, 4)) * 2.0 ** rng.integers(-12, 3, (200, 4))
    c = rng.uniform(-1, 1, (200, 1))
    even = np.concatenate([h[:, ::-1], c, h], axis=1)
    odd = np.concatenate([-h[:, ::-1], 0.0 * c, h], axis=1)
    assert np.all(run(even, scheme, 0) == 0.0) and np.all(run(even, scheme, 1) == 0.0)
    assert np.all(run(odd, scheme, 2) == 0.0)
    for nD in (2, 3):
        axes = np.stack([np.roll(odd, k, axis=0) * [1.0, -1.0, 3.0][k] for k in range(nD)], axis=1)
        axes[:, :, 4] = 0.0
        assert np.all(run_groups(boxes(axes), len(axes), scheme, nD) == 0.0)
    signed = np.array([1.0, -0.0, 2.0, -0.0, 0.0, 0.0, 2.0, 0.0, 1.0])
    w = np.stack([signed, signed[::-1], -signed])
    assert np.all(run(w, scheme, 0) == 0.0) and np.all(run(w, scheme, 1) == 0.0)
