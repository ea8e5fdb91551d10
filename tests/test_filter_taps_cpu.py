"""The FP32 taps of the mixed filter's correction F - I (`balance_taps`,
csrc/cs3d_abi.cu, compiled for the host): like the exact ones they leave a
constant alone, and the largest scales but for the square of their wavenumber."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from test_seq_tasks_cpu import CSRC, SHIM, _between

MAIN = r"""
#include <cmath>
#include <cstring>
#include <vector>
#include "cs3d.h"
#include "cs3d_dev.cuh"
using namespace cs3d;
namespace cs3d { struct SeqOp; struct WallOp; }
namespace {
@HOST@
}
// FP32 taps, the recurrence's coefficient, and the correction's gain at wavenumber k
extern "C" double taps(double alphaF, double k, float *out, double *nl) {
    const HostOp F = make_op(3, 128, CS3D_PERIODIC_SOLVE, 1.0, alphaF), c = make_filter_correction(F);
    const SegPlan p = seg_plan(128, false);
    SegOp<float> o = seg_op<float>(c, p);
    balance_taps(seg_op<double>(c, p).s, o.s);
    for (int h = 0; h <= kMaxH; h++) out[h] = o.s[h];
    *nl = o.nl;
    // (the exact symbol of the order eight filter's numerator: a multiple of (1 - cos k)^4)
    return -(1.0 - 2.0 * alphaF) / 16.0 * std::pow(1.0 - std::cos(k), 4) / (1.0 + 2.0 * alphaF * std::cos(k));
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("taps")
    abi = open(os.path.join(CSRC, "cs3d_abi.cu")).read()
    host = (_between(abi, "struct HostOp {", "// Device copy of an operator")
            + _between(abi, "// How a periodic line of N points is cut", "// Whether the left-hand side (a, 1, a) factors"))
    (d / "cuda_runtime.h").write_text(SHIM)
    (d / "main.cpp").write_text(MAIN.replace("@HOST@", host))
    so = d / "taps.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-w", "-I", str(d), "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), str(d / "main.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.taps.argtypes = [ctypes.c_double, ctypes.c_double, ctypes.POINTER(ctypes.c_float),
                         ctypes.POINTER(ctypes.c_double)]
    lib.taps.restype = ctypes.c_double
    return lib


@pytest.mark.parametrize("alphaF", [0.49, 0.495, 0.48, 0.47, 0.45, 0.4, 0.3, 0.1, 0.0, -0.2, -0.45])
def test_large_scales_are_left_alone(lib, alphaF):
    for m in (1, 2, 3, 4):
        k = 2.0 * np.pi * m / 128
        s, nl = np.zeros(5, np.float32), ctypes.c_double()
        exact = lib.taps(alphaF, k, s.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), ctypes.byref(nl))
        t = s.astype(np.float64)
        assert t[0] + 2.0 * t[1:].sum() == 0.0
        lhs = abs(1.0 - nl.value * np.exp(-1j * k)) ** 2
        gain = (t[0] + 2.0 * (t[1:] * np.cos(np.arange(1, 5) * k)).sum()) / lhs
        # one unit of the taps times k^2 (each tap is within one and a half units, and
        # their second moment was made least)
        assert abs(gain - exact) <= np.spacing(s[1:3]).max() * k * k / lhs
