// cs3d_dev.cuh -- device-side data structures and helpers shared by the
// kernels and the host set-up code of the GB300 stage path.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace cs3d {

// Maximum half width of a compact stencil's right-hand side: 2 for the
// derivatives (Derivatives.cpp:119-247), 4 for the filter (Filter.cpp:5-96).
constexpr int kMaxH = 4;
constexpr int kTaps = 2 * kMaxH + 1;

// One compact operator along one direction with its Thomas factors
// precomputed on the host.  The reference re-derives the factors, the
// Sherman-Morrison vector z and every division on every line of every call
// (Utils.cpp:4-46); here they are computed once per solver, so a line solve
// is one multiply-add forward and one multiply-add plus multiply backward.
//
//   forward   y_0 = r_0,  y_n = r_n - m_n y_{n-1}
//   backward  x_{N-1} = y_{N-1} iw_{N-1},  x_n = (y_n - c_n x_{n+1}) iw_n
//   cyclic    x_n -= f z_n,   f = (x_0 + bog x_{N-1}) inv_den   (f in FP64)
constexpr int kU = 4;  // rows per unrolled chunk of the line solves

template <typename T>
struct LineOp {
    const T *m;          // forward multipliers a_n / w_{n-1}        [N]
    const T *iw;         // reciprocals of the eliminated diagonal    [N]
    const T *c;          // super-diagonal                           [N]
    const T *z;          // Sherman-Morrison vector (periodic only)   [N]
    const T *mf;         // m from row H on: mf[k] = m[H+k]  (chunked forward loads)
    const T *cbk;        // c backwards: cbk[k] = c[N-2-k]   (chunked backward loads)
    const T *ibk;        // iw backwards: ibk[k] = iw[N-2-k]
    T taps[kTaps];       // interior RHS stencil, centred at kMaxH
    T btaps[2 * kMaxH][kTaps]; // the first H and last H rows, explicit
    int boff[2 * kMaxH]; // first column of each boundary row
    T scale;             // 1/h, 1/h^2 or 1
    // Rows [klo, khi) (kU <= klo, khi <= N-1) where m, iw and c equal km,
    // kiw, kc bit for bit in T: the factors of the Toeplitz interior converge
    // geometrically, and there the recurrences run on register constants.
    T km, kiw, kc;
    int klo, khi;
    double bog;          // beta / gamma of the cyclic correction
    double inv_den;      // 1 / (1 + z_0 + beta z_{N-1} / gamma)
    int N;
    int H;               // stencil half width (2 or 4)
    int periodic;
};

constexpr int kSeqSeg = 64;  // SegPlan::SEG of the plain form's sequential solves

// How a periodic line is cut into register segments (cs3d_seg.cuh): G
// segments (a power of two, one lane each), the first nS of S rows and the
// others of S - 1, walked by a kernel compiled for SEG rows a segment.
struct SegPlan {
    int SEG;   // 0: not cut (the Thomas solves run instead)
    int full;  // every segment has SEG rows
    int S, nS, G;
    int lgLW;  // log2 of the lines a warp holds: 32 / G
    int pad;   // full only: shared-memory elements between a line's segments
    int kS;    // SEG - S
    int pair;  // array elements are float2 (y and z sweeps), else float
    int wall;  // cluster: a line between walls (WallOp)
    int C, B;  // C > 0: a cluster of C blocks holds the line, B segments each
               // (G = B C, not restricted to a power of two)
};

// A periodic operator in that form: -l, the scaled taps (centre outwards; second derivative: seg_r2),
// the powers (-l)^(k+1), and what weights the carries between segments.
template <typename R>
struct SegOp {
    R nl, s[kMaxH + 1], pw[32];
    R qS, qS1;  // (-l)^S, (-l)^(S-1)
    R iS, iS1;  // (-l)^-kS, (-l)^-(kS+1)
    R geo;          // 1 / (1 - l^2)
    R wrap;     // 1, or 1 / (1 - (-l)^N) where T = G
    int T;
};

// Loads of operator coefficients (a few kB per operator, read by every line
// solve) through the read-only data path.
__device__ __forceinline__ float ldc(const float *p) { return __ldg(p); }
__device__ __forceinline__ double ldc(const double *p) { return __ldg(p); }

// Four consecutive coefficients from a 16-byte aligned address in one or two
// 128-bit loads.
__device__ __forceinline__ void load4(const float *p, float v[4]) {
    const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void load4(const double *p, double v[4]) {
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldg(reinterpret_cast<const double2 *>(p + 2));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// Conserved variables of one state (five FP64 arrays, XYZ layout).
struct Q5 {
    double *f[5];
};

// Division by a fixed d > 0 of numerators below 2^31:
// p / d = (umulhi(p, mul) + p) >> sh  (Granlund-Montgomery, round-up form).
struct FastDiv {
    unsigned mul;
    int sh;
};

inline FastDiv make_fastdiv(unsigned d) {
    FastDiv f;
    int sh = 0;
    while ((1ull << sh) < d) ++sh;
    f.sh = sh;
    f.mul = (unsigned)((((1ull << 32) * ((1ull << sh) - d)) / d) + 1ull);
    return f;
}

// Grid geometry.
struct Geom {
    int Nx, Ny, Nz;
    long long npts;
};

// ---------------------------------------------------------------------
// FP32 <-> FP64 conversion with integer instructions.  On this part the
// hardware conversions issue on the FP64 pipe, which runs at 1/64 of the
// FP32 rate; these take a handful of integer operations instead.  Both follow
// the IEEE-754 binary32/binary64 layouts: exact widening, and narrowing with
// round-to-nearest-even.  Subnormal results are flushed to signed zero and
// values beyond the binary32 range become infinity (NaN as well), which is
// immaterial for a flow state and its increments.
// ---------------------------------------------------------------------
__device__ __forceinline__ double widen(float f) {
    const unsigned u = __float_as_uint(f);
    const unsigned sign = u & 0x80000000u;
    const unsigned ex = (u >> 23) & 0xffu;
    const unsigned man = ex == 0u ? 0u : (u & 0x7fffffu);
    const unsigned e64 = ex == 0u ? 0u : (ex == 0xffu ? 0x7ffu : ex + 896u);
    const unsigned hi = sign | (e64 << 20) | (man >> 3);
    const unsigned lo = man << 29;
    return __hiloint2double((int)hi, (int)lo);
}

__device__ __forceinline__ float narrow(double d) {
    const unsigned hi = (unsigned)__double2hiint(d);
    const unsigned lo = (unsigned)__double2loint(d);
    const unsigned sign = hi & 0x80000000u;
    const int ex = (int)((hi >> 20) & 0x7ffu);
    const int e32 = ex - 896;
    const unsigned m = ((hi & 0xfffffu) << 3) | (lo >> 29);
    const unsigned rest = lo & 0x1fffffffu;
    unsigned bits = ((unsigned)e32 << 23) + m;
    bits += (rest > 0x10000000u) | ((rest == 0x10000000u) & (m & 1u));
    bits = e32 <= 0 ? 0u : (e32 >= 255 ? 0x7f800000u : bits);
    bits = bits > 0x7f800000u ? 0x7f800000u : bits;
    return __uint_as_float(sign | bits);
}

// d as the unevaluated sum of two floats: hi its leading 24 bits, lo the next
// 23, by integer instructions.  |d| below 2^-70 (or not finite): hi alone.
__device__ __forceinline__ void split(double d, float &hi, float &lo) {
    const unsigned h = (unsigned)__double2hiint(d), l = (unsigned)__double2loint(d);
    const unsigned sign = h & 0x80000000u;
    const int e32 = (int)((h >> 20) & 0x7ffu) - 896;
    // truncated, so that the low 29 mantissa bits are the remainder
    unsigned b = ((unsigned)e32 << 23) | ((h & 0xfffffu) << 3) | (l >> 29);
    b = e32 <= 0 ? 0u : (e32 >= 255 ? 0x7f800000u : b);
    hi = __uint_as_float(sign | b);
    // the upper 23 of them as a float in [0, 1) ulp of hi
    const float r = __uint_as_float(0x3f800000u | ((l >> 6) & 0x7fffffu)) - 1.0f;
    const bool small = e32 <= 57 || e32 >= 255;
    lo = small ? 0.0f : r * __uint_as_float(sign | ((unsigned)(e32 - 23) << 23));
}

// q - ref in FP32 (ref = ref_hi + ref_lo): both parts' differences, each exact
// or rounded relative to the result.  An FP64 subtraction here would double
// the last stage's work on the FP64 pipe.
__device__ __forceinline__ float fluct_of(double q, float ref_hi, float ref_lo) {
    float hi, lo;
    split(q, hi, lo);
    return (hi - ref_hi) + (lo - ref_lo);
}

// Work-precision <-> FP64 without the FP64 conversion pipe.
template <typename T> __device__ __forceinline__ T to_work(double d);
template <> __device__ __forceinline__ double to_work<double>(double d) { return d; }
template <> __device__ __forceinline__ float to_work<float>(double d) { return narrow(d); }
__device__ __forceinline__ double to_f64(double x) { return x; }
__device__ __forceinline__ double to_f64(float x) { return widen(x); }

// Bit f set if point (i,j,k) lies on face f (X0,X1,Y0,Y1,Z0,Z1).
__device__ __forceinline__ int faces_of(const Geom &g, int i, int j, int k) {
    int f = 0;
    f |= (i == 0) << 0; f |= (i == g.Nx - 1) << 1;
    f |= (j == 0) << 2; f |= (j == g.Ny - 1) << 3;
    f |= (k == 0) << 4; f |= (k == g.Nz - 1) << 5;
    return f;
}

// Reciprocal and square root in FP64 from FP32 estimates by one step of a
// cubically convergent Newton series (1/x = r (1 + e + e^2 + ...), e = 1 - x r;
// sqrt x = g (1 - e)^(-1/2), g = x r, e = 1 - g r with r near 1/sqrt x): three and
// five operations on the FP64 pipe, within an ulp (the square root: one and a
// half).  Outside the FP32 range, and for NaN, the library's.
__device__ __forceinline__ double rcp_f64(double x) {
    if (!(fabs(x) > 1e-30 && fabs(x) < 1e30)) return 1.0 / x;
    const double r = widen(__frcp_rn(narrow(x)));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double sqrt_f64(double x) {
    if (!(x > 1e-30 && x < 1e30)) return sqrt(x);
    const double r = widen(__frsqrt_rn(narrow(x))), g = x * r;
    const double e = fma(-g, r, 1.0);
    return fma(g * e, fma(0.375, e, 0.5), g);
}

// a / b in FP32 from ib, b's hardware reciprocal (rcp_est, one ulp): the
// product's residual, exact by FMA, corrects it (Markstein, IBM J. Res. Dev. 34,
// 1990), to within a few thousandths of an ulp of the rounded quotient.  Several
// quotients of one b share the reciprocal; b must be normal.
__device__ __forceinline__ float rcp_est(float b) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    return r;
}
__device__ __forceinline__ float quot(float a, float b, float ib) {
    const float q = a * ib;
    return fmaf(fmaf(-q, b, a), ib, q);
}

// T^-0.24 and T^0.76, for the viscosity law mu = mu_ref T^0.76 (IdealGas.hpp)
// and its slope 0.76 mu / T = 0.76 mu_ref T^-0.24.
// FP32: exp2(-0.24 log2 T) with the hardware log2 (absolute error about 2^-22,
// so about 4e-8 relative in the result), and T times that.
__device__ __forceinline__ float visc_rpow(float T) { return exp2f(-0.24f * __log2f(T)); }
__device__ __forceinline__ float visc_pow(float T) { return T * visc_rpow(T); }
// FP64, whose pipe issues two operations per SM and clock: y = T^-0.24 solves
// T^6 y^25 = 1; from an FP32 estimate (relative error below 6e-7) the residual
// e = 1 - T^6 y^25 gives the factor (1 - e)^(-1/25) = 1 + e/25 + 13 e^2/625 + ...,
// the next term below 5e-17, of both powers.  T^0.76 is T y with the rounding
// of that product and the factor's excess added: as T times T^-0.24 it had two
// roundings more (1.8 ulp at most, 0.9 so; three FP64 operations more, as many as
// (T y^4)^6 y takes less than T^6 times y^25).  No division; both within 1.3 ulp
// on [1e-6, 1e6], 1.0 near T = 1.  Outside that range, and for NaN, the library
// pow.
__device__ __forceinline__ double visc_powers(double T, double &rpow) {
    if (!(T > 1e-6 && T < 1e6)) {
        rpow = pow(T, -0.24);
        return pow(T, 0.76);
    }
    const double y = widen(exp2f(-0.24f * log2f(narrow(T)))), ty = T * y;
    const double y2 = y * y, u = T * (y2 * y2), u2 = u * u;  // (T y^4)^6 y
    const double e = fma(-(u2 * u2 * u2), y, 1.0);
    const double g = e * fma(e, 13.0 / 625.0, 1.0 / 25.0);
    rpow = fma(y, g, y);
    return ty + fma(ty, g, fma(T, y, -ty));
}
__device__ __forceinline__ double visc_pow(double T) {
    double r;
    return visc_powers(T, r);
}
__device__ __forceinline__ double visc_rpow(double T) {
    double r;
    visc_powers(T, r);
    return r;
}

// Direction whose continuity derivative survives at a wall point: the
// reference applies the wall faces in the order X0,X1,Y0,Y1,Z0,Z1 and the
// last write wins (CSolver_AWS.cpp:1526-1609).  -1 if not on a wall.
__device__ __forceinline__ int wall_dir(int onwall) {
    return (onwall & 0x30) ? 2 : (onwall & 0x0c) ? 1 : (onwall & 0x03) ? 0 : -1;
}

}  // namespace cs3d
