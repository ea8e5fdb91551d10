"""The mixed form's FP32 quotient (`quot`, csrc/cs3d_dev.cuh) restated in numpy:
a product with a reciprocal of up to one ulp error, corrected by its residual.
Each FP32 operation is a float64 one rounded to float32 (products of two floats
are exact in float64, so the fused steps are too)."""
import numpy as np


def test_within_one_ulp_of_the_rounded_quotient():
    rng = np.random.default_rng(3)
    n = 400_000
    f32 = np.float32
    a = (rng.standard_normal(n) * 10.0 ** rng.uniform(-3, 3, n)).astype(f32)
    b = (10.0 ** rng.uniform(-3, 3, n)).astype(f32)
    exact = a.astype(np.float64) / b.astype(np.float64)
    for off in (-1, 0, 1):  # the reciprocal's last place
        ib = (1.0 / b.astype(np.float64)).astype(f32)
        ib = np.nextafter(ib, f32(np.inf) if off > 0 else f32(0)) if off else ib
        q = (a.astype(np.float64) * ib).astype(f32)
        e = (a.astype(np.float64) - q.astype(np.float64) * b).astype(f32)
        r = (e.astype(np.float64) * ib + q).astype(f32)
        ulps = np.abs(r.astype(np.float64) - exact) / np.spacing(np.abs(exact).astype(f32))
        assert ulps.max() <= 0.51
