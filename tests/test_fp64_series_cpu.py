"""The FP64 reciprocal, square root and viscosity power T^-0.24 of the kernels
(`rcp_f64`, `sqrt_f64`, `visc_rpow`, csrc/cs3d_dev.cuh) restated in numpy: an
FP32 estimate and one step of a cubically convergent series.  Fused steps are
formed in long double and rounded."""
import numpy as np

LD = np.longdouble


def _ulps(r, ref):
    return np.abs(r.astype(LD) - ref) / np.spacing(np.abs(ref).astype(np.float64))


def _fma(a, b, c):
    return (a.astype(LD) * b + c).astype(np.float64)


def _sample(lo, hi):
    return 10.0 ** np.random.default_rng(5).uniform(lo, hi, 400_000)


def test_reciprocal_within_an_ulp():
    # the estimate is off by e below 2^-23 (x and 1/x rounded to FP32), the next
    # term of the series is e^3 = 2^-69; two roundings of half an ulp
    x = _sample(-29, 29)
    r = (1.0 / x.astype(np.float32)).astype(np.float32).astype(np.float64)
    e = _fma(-x, r, 1.0)
    y = _fma(r, _fma(e, e, e), r)
    assert _ulps(y, LD(1) / x).max() <= 1.0


def test_square_root_within_an_ulp():
    x = _sample(-29, 29)
    r = (1.0 / np.sqrt(x.astype(np.float32).astype(np.float64))).astype(np.float32).astype(np.float64)
    g = x * r
    e = _fma(-g, r, 1.0)
    y = _fma(g * e, _fma(np.full_like(e, 0.375), e, 0.5), g)
    # g's rounding (half an ulp) survives, as sqrt x = g (1 - e)^(-1/2) holds
    # for the exact g: with the final one, one ulp
    assert _ulps(y, np.sqrt(x.astype(LD))).max() <= 1.5


def test_viscosity_power_within_two_ulp():
    # rounding of T^6 (5 half ulps) and y^25 (24) reaches y divided by 25: 1.2,
    # and one of the last step: 1.1 ulp, and the neglected term 5e-17
    T = _sample(-6, 6)
    y = np.exp2(np.float32(-0.24) * np.log2(T.astype(np.float32))).astype(np.float64)
    t2 = T * T
    t6 = t2 * t2 * t2
    y2 = y * y
    y4 = y2 * y2
    y8 = y4 * y4
    y16 = y8 * y8
    e = _fma(-t6, y16 * y8 * y, 1.0)
    r = _fma(y, e * _fma(e, np.full_like(e, 13.0 / 625.0), 1.0 / 25.0), y)
    assert _ulps(r, T.astype(LD) ** LD(-0.24)).max() <= 2.0
