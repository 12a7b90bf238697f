"""The quotients of the block-interface SATs' Roe average and unit normal, plain
and on dual numbers, are rounded once: bitwise the same expressions in numpy
(host build of the device functions, without contraction)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from magudi_gb300 import build, capi

SOURCE = r'''
#include <cuda_runtime.h>
#include "mgd_device.cuh"
using namespace mgd;
template <int ND> static void average(const double* qL, const double* qR, const double* m, double g, double* out) {
  constexpr int nU = ND + 2;
  typedef DualN<1> D;
  double roe[nU];
  roeAverage<ND, double, double>(qL, qR, g, roe);
  D dL[nU], dual[nU];
  for (int c = 0; c < nU; ++c) dL[c] = D(qL[c]), dL[c].d[0] = 1.0;
  roeAverage<ND, D, double>(dL, qR, g, dual);
  const Incoming<ND, double> I = incomingState<ND, double>(roe, m, g, 1);
  for (int c = 0; c < nU; ++c) out[c] = roe[c], out[nU + c] = dual[c].v;
  for (int d = 0; d < ND; ++d) out[2 * nU + d] = I.n[d];
}
extern "C" void averages(int nD, int n, const double* qL, const double* qR, const double* m, double g, double* out) {
  for (int s = 0; s < n; ++s) {
    if (nD == 2) average<2>(qL + 4 * s, qR + 4 * s, m + 2 * s, g, out + 10 * s);
    else average<3>(qL + 5 * s, qR + 5 * s, m + 3 * s, g, out + 13 * s);
  }
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotients")
    src, so = d / "q.cu", d / "libq.so"
    src.write_text(SOURCE)
    subprocess.check_call([build.nvcc(), *build.ARCH_FLAGS, "-std=c++17", "-O2", "-w", "-I", build.CSRC, "-shared",
                           "-Xcompiler", "-fPIC", "-Xcompiler", "-ffp-contract=off", str(src), "-o", str(so)],
                          env=dict(os.environ, TMPDIR=str(d)))
    return C.CDLL(str(so))


@pytest.mark.parametrize("nD", [2, 3])
def test_roe_average_and_normal_are_rounded_once(lib, nD):
    rng = np.random.default_rng(21)
    n, nU, g = 500, nD + 2, 1.4

    def states():
        rho, u = rng.uniform(0.5, 2.0, n), rng.uniform(-1, 1, (n, nD))
        E = rng.uniform(0.4, 1.2, n) / (g - 1.0) + 0.5 * rho * np.sum(u * u, axis=1)
        return np.ascontiguousarray(np.column_stack([rho, rho[:, None] * u, E]))

    qL, qR, m = states(), states(), np.ascontiguousarray(rng.uniform(-2, 2, (n, nD)))
    out = np.zeros((n, 2 * nU + nD))
    lib.averages(nD, n, capi.dptr(qL), capi.dptr(qR), capi.dptr(m), C.c_double(g), capi.dptr(out))

    def sum_of_squares(v):
        s = v[0] * v[0]
        for t in v[1:]:
            s = s + t * t
        return s

    L, R = qL.T, qR.T
    sL, sR = np.sqrt(L[0]), np.sqrt(R[0])
    h = [g * q[-1] - 0.5 * (g - 1.0) * (1.0 / q[0]) * sum_of_squares(q[1:-1]) for q in (L, R)]
    roe = [sL * sR] + [(sR * L[1 + d] + sL * R[1 + d]) / (sL + sR) for d in range(nD)]
    e = (sR * h[0] + sL * h[1]) / (sL + sR)
    roe.append((e + 0.5 * (g - 1.0) / roe[0] * sum_of_squares(roe[1:])) / g)
    arc = np.sqrt(sum_of_squares(m.T))
    assert np.array_equal(out[:, :nU].T, np.array(roe))
    assert np.array_equal(out[:, nU:2 * nU].T, np.array(roe))
    assert np.array_equal(out[:, 2 * nU:].T, m.T / arc)
