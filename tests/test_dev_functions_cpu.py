"""The device functions of csrc/cs3d_dev.cuh compiled for the host, against
long double: the FP64 viscosity powers, reciprocal and square root from FP32
estimates."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from test_seq_tasks_cpu import SHIM

CSRC = os.path.join(ROOT, "3dcompactsolver_gb300", "csrc")

MAIN = r"""
#include "cs3d_dev.cuh"
using namespace cs3d;
// errors in units of the last place of the exact value
static double ulps(double r, long double x) {
    const double a = (double)fabsl(x);
    return (double)(fabsl(r - x) / (nextafter(a, 1e308) - a));
}
extern "C" double visc076(double T) { return ulps(visc_pow(T), powl(T, 0.76L)); }
extern "C" double visc024(double T) { return ulps(visc_rpow(T), powl(T, -0.24L)); }
extern "C" double reciprocal(double x) { return ulps(rcp_f64(x), 1.0L / x); }
extern "C" double root(double x) { return ulps(sqrt_f64(x), sqrtl(x)); }
"""


@pytest.fixture(scope="module")
def dev(tmp_path_factory):
    d = tmp_path_factory.mktemp("dev")
    (d / "cuda_runtime.h").write_text(SHIM)
    (d / "main.cpp").write_text(MAIN)
    so = d / "dev.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-w", "-I", str(d), "-I", CSRC,
                    str(d / "main.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    for f in ("visc076", "visc024", "reciprocal", "root"):
        getattr(lib, f).argtypes = [ctypes.c_double]
        getattr(lib, f).restype = ctypes.c_double
    return lib


def _worst(f, lo, hi, n=60_000):
    return max(f(float(x)) for x in 10.0 ** np.random.default_rng(7).uniform(lo, hi, n))


# In units u = 2^-53, at most a last place each.  (T y^4)^6 carries 8.5 u (y having
# 24 bits, y^2 is exact: 1 in T y^4, 2.5 in its square, 8.5 in that one's cube),
# divided by 25 in the powers: 0.34; the last addition 0.5; the series' next term
# 0.43 at the estimate's worst, none near T = 1.
@pytest.mark.parametrize("f", ["visc076", "visc024"])
@pytest.mark.parametrize("lo,hi,bound", [(-6, 6, 1.3), (-1, 1, 1.0)])
def test_viscosity_powers(dev, f, lo, hi, bound):
    assert _worst(getattr(dev, f), lo, hi) <= bound


@pytest.mark.parametrize("f,bound", [("reciprocal", 1.0), ("root", 1.5)])
def test_reciprocal_and_root(dev, f, bound):
    assert _worst(getattr(dev, f), -29, 29) <= bound
