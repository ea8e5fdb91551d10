// cs3d_lineop.cu -- one compact operator on contiguous FP64 lines
// (Derivatives::calc1stDerivField, calc2ndDerivField, Filter::filterField) in
// register segments (sm_103a).
//
// A warp owns 32 / G whole lines, G segments each, one segment a lane: it
// copies its lines (one contiguous range of memory) to its own shared memory,
// every lane solves its segment in registers (cs3d_seg.cuh), and the warp copies
// the result out.  Nothing is shared between warps, so loads, solves and
// stores of different warps overlap without block barriers.  Segments are
// SEG + 1 doubles apart: 32 lanes at the same row touch all banks.
//
// What bounds it: FP64 issue (two operations an SM and clock).  The kernel it
// replaces on these lengths (k_line_op: one thread a line, a quarter of the
// block's threads) left that pipe idle most of the time: 128^3, three operators,
// 235 us; walls of 301 points (3850 lines), 161 us.
#include "cs3d_seg.cuh"
#include "cs3d_kernels.cuh"

namespace cs3d {

constexpr int kLineSegTpb = 128;

extern __shared__ __align__(16) unsigned char smem_line[];

// The solve of a line with wall closures: the factors vary along the line, so
// each row's come from a table (SegTab), walked like the registers.
template <int SEG>
__device__ __forceinline__ void seg_solve_tab(double (&y)[SEG], const SegTab &tb, int T, int G, int seg, int k0,
                                              int lane0) {
    const double *f = tb.f + seg * SEG, *b = tb.b + seg * SEG, *pf = tb.pf + seg * SEG, *pb = tb.pb + seg * SEG;
    double c = 0.0;
#pragma unroll
    for (int k = 0; k < SEG; ++k) y[k] = c = fma(ldc(f + k), c, y[k]);
    double in = 0.0, q = ldc(pf + SEG - 1);
    for (int t = T; t >= 1; --t) {
        const int src = max(seg - t, 0);
        const double es = __shfl_sync(0xffffffffu, c, lane0 + src), qs = __shfl_sync(0xffffffffu, q, lane0 + src);
        in = seg - t >= 0 ? fma(qs, in, es) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < SEG; ++k) y[k] = fma(ldc(pf + k), in, y[k]);
    c = 0.0;
    double first = 0.0;
#pragma unroll
    for (int k = SEG - 1; k >= 0; --k) {
        y[k] = c = fma(ldc(b + k), c, y[k]);
        if (k <= kSegSlack) first = k == k0 ? c : first;
    }
    in = 0.0;
    q = ldc(pb + k0);
    for (int t = T; t >= 1; --t) {
        const int src = min(seg + t, G - 1);
        const double es = __shfl_sync(0xffffffffu, first, lane0 + src), qs = __shfl_sync(0xffffffffu, q, lane0 + src);
        in = seg + t < G ? fma(qs, in, es) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < SEG; ++k) y[k] = fma(ldc(pb + k), in, y[k]);
}

// KIND 1, 2: derivatives, 3: filter.  WALL: closures from op's explicit rows
// and factors from a.tab; else periodic.
template <int KIND, int SEG, bool FULL, bool WALL>
__global__ void __launch_bounds__(kLineSegTpb, WALL && SEG > 24 ? 3 : 4) k_line_seg(LineSegArgs a) {
    constexpr int H = KIND == 3 ? 4 : 2, LS = SEG + 1;
    const int N = a.N, G = a.seg.G, lane = threadIdx.x & 31, lw = 32 >> a.lgG;
    const long long l0 = ((long long)blockIdx.x * (kLineSegTpb / 32) + (threadIdx.x >> 5)) * lw;
    if (l0 >= a.nlines) return;  // (whole warps)
    const int total = (int)min((long long)lw, a.nlines - l0) * N;
    double *sm = reinterpret_cast<double *>(smem_line) + (threadIdx.x >> 5) * 32 * LS;
    const int nb = a.seg.nS * a.seg.S;
    // shared-memory offset of the warp's element idx
    auto place = [&](int idx) {
        const int l = (int)((__umulhi((unsigned)idx, a.divN.mul) + (unsigned)idx) >> a.divN.sh), n = idx - l * N;
        int seg, k;
        if (FULL) {
            seg = n / SEG;
            k = n % SEG;
        } else {
            const bool lng = n < nb;
            const FastDiv d = lng ? a.divS : a.divS1;
            const int m = lng ? n : n - nb, s = (int)((__umulhi((unsigned)m, d.mul) + (unsigned)m) >> d.sh);
            seg = lng ? s : s + a.seg.nS;
            k = m - s * (lng ? a.seg.S : a.seg.S - 1);
        }
        return ((l << a.lgG) + seg) * LS + k;
    };
    const double *in = a.in + l0 * N;
    for (int i0 = lane; i0 < total; i0 += 8 * 32) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = i0 + 32 * u < total ? in[i0 + 32 * u] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (i0 + 32 * u < total) sm[place(i0 + 32 * u)] = v[u];
    }
    __syncwarp();
    const int seg = lane & (G - 1), lane0 = lane & ~(G - 1);
    const int len = a.seg.S - (seg >= a.seg.nS), k0 = SEG - len;
    const int sp = (seg - 1) & (G - 1), sn = (seg + 1) & (G - 1);
    SegLane<double> s;
    s.seg = seg;
    s.k0 = k0;
    s.row = sm + lane * LS - k0;
    s.lo = sm + (lane0 + sp) * LS + a.seg.S - (sp >= a.seg.nS) - k0;
    s.hi = sm + (lane0 + sn) * LS;
    double y[SEG];
    {
        double w[SEG + 2 * H];
        seg_load<SEG, FULL, H>(w, s, 1, [](const double *p) { return *p; });
#pragma unroll
        for (int k = 0; k < SEG; ++k) {
            if constexpr (KIND == 1) y[k] = seg_r1<SEG>(w, a.op, k);
            if constexpr (KIND == 2) y[k] = seg_r2<SEG>(w, a.op, k);
            if constexpr (KIND == 3) y[k] = seg_r3<SEG>(w, a.op, k);
            if (!FULL && k < kSegSlack && k < k0) y[k] = 0.0;
        }
    }
    if constexpr (WALL) {
        // the first and last H rows, from their explicit coefficients
        // (their columns lie in the line's first or last two segments).  A derivative's
        // sum to zero: differences from the wall value, so that their rounding makes
        // no derivative of a constant.  It was most of the second derivative's error: 301
        // points 1.0e-13 of the result, so 1.8e-14.
        const double *line0 = sm + lane0 * LS;
        auto explicit_row = [&](int r, int sa, double base) {
            const int na = seg_row0(a.seg, sa), nb2 = seg_row0(a.seg, min(sa + 1, G - 1));
            const double *pa = line0 + sa * LS - na, *pb = line0 + min(sa + 1, G - 1) * LS - nb2;
            double v = 0.0;
            for (int k = 0; k < (KIND == 3 ? 7 : 6); ++k) {  // (no wall row has more columns)
                const int n = a.boff[r] + k;
                if (n >= N) break;
                const double x = n >= nb2 ? pb[n] : pa[n];
                v = fma(a.btaps[r][k], KIND == 3 ? x : x - base, v);
            }
            return v;
        };
        if (seg == 0 || seg == G - 1) {
            const double wall = KIND == 3 ? 0.0 : s.row[seg == 0 ? k0 : SEG - 1];
#pragma unroll
            for (int b = 0; b < H; ++b) {
                const double v = explicit_row(seg == 0 ? b : H + b, seg == 0 ? 0 : max(G - 2, 0), wall);
                // (selects: as an assignment to row k0 + b the array leaves the
                // registers)
                const bool lo = seg == 0;
#pragma unroll
                for (int k = 0; k < kSegSlack + H; ++k) y[k] = lo && k == k0 + b ? v : y[k];
                y[SEG - H + b] = lo ? y[SEG - H + b] : v;
                if (G == 1) y[SEG - H + b] = explicit_row(H + b, 0, s.row[SEG - 1]);
            }
        }
        const double *sc = a.tab.s + seg * SEG;
#pragma unroll
        for (int k = 0; k < SEG; ++k) y[k] *= ldc(sc + k);
        seg_solve_tab<SEG>(y, a.tab, a.op.T, G, seg, k0, lane0);
    } else {
        // 64 bits: the second derivative's powers fall below 1e-17 in 24 rows
        seg_solve<SEG, FULL, (KIND == 2 ? 24 : SEG)>(y, a.op, a.seg, seg, k0, lane0, 0);
    }
    __syncwarp();  // every lane has read its window
    seg_store<SEG, FULL>(s, 1, [&](double *p, int k) { *p = y[k]; });
    __syncwarp();
    double *out = a.out + l0 * N;
#pragma unroll 8
    for (int i = lane; i < total; i += 32) out[i] = sm[place(i)];
}

// First derivatives along y or z of fields in XYZ layout (periodic lines): a
// lane's rows go from memory to registers and back, with no shared memory.  A
// warp's 32 / G lines are adjacent in x, as are a block's warps.
template <int SEG, bool FULL>
__global__ void __launch_bounds__(kLineSegTpb, 4) k_column_seg(ColumnArgs a) {
    const int G = a.seg.G, lane = threadIdx.x & 31, lw = 32 >> a.lgG;
    const int l = lane & (lw - 1), seg = lane >> (5 - a.lgG);
    const int i0 = ((int)blockIdx.x * (kLineSegTpb / 32) + (int)(threadIdx.x >> 5)) * lw;
    if (i0 >= a.Nx) return;  // (whole warps)
    const int i = min(i0 + l, a.Nx - 1);
    const long long st = a.stride;
    const long long base = (long long)blockIdx.y * a.plane + i;
    const int n0 = seg_row0(a.seg, seg), len = a.seg.S - (seg >= a.seg.nS), k0 = SEG - len;
    const double *src = a.src[blockIdx.z] + base;
    SegLane<const double> s;
    s.seg = seg;
    s.k0 = k0;
    s.row = src + (n0 - k0) * st;
    s.lo = n0 > 0 ? s.row : s.row + a.N * st;
    s.hi = seg < G - 1 ? src + (n0 + len) * st : src;
    double y[SEG];
    {
        double w[SEG + 4];
        seg_load<SEG, FULL, 2>(w, s, st, [](const double *p) { return __ldg(p); });
#pragma unroll
        for (int k = 0; k < SEG; ++k) {
            y[k] = seg_r1<SEG>(w, a.op, k);
            if (!FULL && k < kSegSlack && k < k0) y[k] = 0.0;
        }
    }
    seg_solve<SEG, FULL, kSegRowsAll>(y, a.op, a.seg, seg, k0, l, 5 - a.lgG);
    if (i0 + l >= a.Nx) return;
    SegLane<double> d;
    d.k0 = k0;
    d.row = a.dst[blockIdx.z] + base + (n0 - k0) * st;
    seg_store<SEG, FULL>(d, st, [&](double *p, int k) { *p = y[k]; });
}

cudaError_t launch_column_seg(const ColumnArgs &a, int planes, cudaStream_t s) {
    const int per = (kLineSegTpb / 32) * (32 >> a.lgG);
    const dim3 grid((a.Nx + per - 1) / per, planes, 3);
    if (a.seg.full) k_column_seg<32, true><<<grid, kLineSegTpb, 0, s>>>(a);
    else if (a.seg.SEG == 32) k_column_seg<32, false><<<grid, kLineSegTpb, 0, s>>>(a);
    else if (a.seg.SEG == 28) k_column_seg<28, false><<<grid, kLineSegTpb, 0, s>>>(a);
    else if (a.seg.SEG == 24) k_column_seg<24, false><<<grid, kLineSegTpb, 0, s>>>(a);
    else if (a.seg.SEG == 20) k_column_seg<20, false><<<grid, kLineSegTpb, 0, s>>>(a);
    else k_column_seg<16, false><<<grid, kLineSegTpb, 0, s>>>(a);
    return cudaGetLastError();
}

template <int KIND, int SEG, bool FULL, bool WALL>
static cudaError_t launch(const LineSegArgs &a, cudaStream_t s) {
    const size_t sm = (size_t)kLineSegTpb * (SEG + 1) * 8;
    const long long per = (kLineSegTpb / 32) * (32 >> a.lgG);
    k_line_seg<KIND, SEG, FULL, WALL><<<(unsigned)((a.nlines + per - 1) / per), kLineSegTpb, sm, s>>>(a);
    return cudaGetLastError();
}
template <int KIND>
static cudaError_t launch_kind(const LineSegArgs &a, cudaStream_t s) {
    if (a.wall) {
        if (a.seg.SEG == 32) return launch<KIND, 32, false, true>(a, s);
        if (a.seg.SEG == 28) return launch<KIND, 28, false, true>(a, s);
        if (a.seg.SEG == 24) return launch<KIND, 24, false, true>(a, s);
        if (a.seg.SEG == 20) return launch<KIND, 20, false, true>(a, s);
        return launch<KIND, 16, false, true>(a, s);
    }
    if (a.seg.full) return launch<KIND, 32, true, false>(a, s);
    if (a.seg.SEG == 32) return launch<KIND, 32, false, false>(a, s);
    if (a.seg.SEG == 28) return launch<KIND, 28, false, false>(a, s);
    if (a.seg.SEG == 24) return launch<KIND, 24, false, false>(a, s);
    if (a.seg.SEG == 20) return launch<KIND, 20, false, false>(a, s);
    return launch<KIND, 16, false, false>(a, s);
}
cudaError_t launch_line_seg(int kind, const LineSegArgs &a, cudaStream_t s) {
    return kind == 1 ? launch_kind<1>(a, s) : kind == 2 ? launch_kind<2>(a, s) : launch_kind<3>(a, s);
}

}  // namespace cs3d
