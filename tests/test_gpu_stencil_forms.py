"""Interior stencils in integer arithmetic: the forms that take several fields
at once."""
import ctypes as C

import numpy as np
import pytest

from magudi_gb300 import capi
from magudi_gb300.solver import load_library
from test_gpu_stencil import KINDS, run, windows

pytestmark = pytest.mark.gpu

SCHEMES = [capi.SBP_48, capi.SBP_12, capi.SBP_24, capi.SBP_36]
FIELDS = {0: 3, 1: 4}


def run_groups(x, n, scheme, form):
    L = load_library()
    L.mgd_selftest_stencil_group.argtypes = [C.POINTER(C.c_double), C.c_int, C.c_int, C.c_int, C.POINTER(C.c_double)]
    out = np.zeros(n * FIELDS.get(form, 1))
    assert L.mgd_selftest_stencil_group(capi.dptr(np.ascontiguousarray(x)), n, scheme, form, capi.dptr(out)) == 0
    return out


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("form", [0, 1])
def test_fields_together_are_bitwise_the_fields_alone(scheme, form):
    """A field's sum does not depend on the other fields': beside ordinary ones
    some leave the integers' range, are at rest or cancel."""
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
    alone = run(x.reshape(-1, 9), scheme, form)
    together = run_groups(x, len(x), scheme, form)
    assert np.array_equal(together.view(np.int64), alone.view(np.int64))
