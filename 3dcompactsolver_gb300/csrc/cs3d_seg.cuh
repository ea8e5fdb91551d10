// cs3d_seg.cuh -- compact line solves of periodic lines in register segments,
// shared by the stage sweeps, the filter and the adjoint kernels.
//
// On a periodic line the compact operators' left-hand side is the circulant
// tridiagonal (a, 1, a), which factors exactly into two first-order
// recurrences with constant coefficients,
//   (a, 1, a) = (1 + l E^-1)(1 + l E) / (1 + l^2),   a = l / (1 + l^2), |l| < 1
// (E the shift by one row), so that with the right-hand side scaled by
// (1 + l^2) -- folded into the taps --
//   forward   y_n = r_n - l y_{n-1},     backward   x_n = y_n - l x_{n+1}
// around the circle.  No row needs factors from memory, a division or a
// Sherman-Morrison correction, and the recurrences are cut anywhere: a line is
// split into G segments, one lane each, held in registers.  Each lane runs its
// segment from a zero start; the value entering it is the ends of the segments
// before it, weighted by powers of -l,
//   Y_j = e_{j-1} + q_{j-1} (e_{j-2} + q_{j-2} (...)),   q = (-l)^length,
// taken from the T nearest segments by shuffles (T: until the weight is below
// 2^-30; the whole circle, with the geometric factor 1 / (1 - (-l)^N), where
// that takes all of them), and is added to the first rows with the same
// powers.  The backward pass mirrors it.
//
// What bounds it: the one-thread-per-line Thomas solve it replaces
// (solve_lanes) was a chain of N rows, each with two shared-memory reads and
// two writes and about 22 instructions, run by half of the block's warps; here
// a row is read once and written once in about 11 instructions, the chain is a
// segment, and a warp holds all segments of its lines (no block barrier inside
// a solve).  The consume phases read solutions without a correction.  Against
// solve_lanes, per step, y and z by the clusters below: 128^3 x 0.250 -> 0.166 ms, y
// 0.358 -> 0.232, z 0.603 -> 0.426; the error against 64 bits falls by a tenth
// (differences before products).
#pragma once
#include "cs3d_dev.cuh"

namespace cs3d {

// FP32: rows at the start of a segment whose carry is added: (-l)^(k+1) falls
// below 5e-9 after these many rows.  The first derivative has l = 0.382, the second
// 0.188; the filter's l depends on its coefficient (all rows).
constexpr int kSegRows1 = 20, kSegRows2 = 12, kSegRowsAll = 64;
// Segments are at most kSegSlack rows shorter than the compiled length (seg_plan keeps
// 8, cluster_plan 12).
constexpr int kSegSlack = 12;

// One lane's place in its line's segments, in elements of the array walked:
// register row k is at row[k * P] (k >= k0), rows before the segment at
// lo[k * P] (k < k0), rows after it at hi[h * P].
template <typename E>
struct SegLane {
    int seg, k0;  // k0: unused leading rows of the register segment
    E *row, *lo, *hi;
};

// First row of segment s, and the rows of segment s (-1: the last).
__device__ __forceinline__ int seg_row0(const SegPlan &pl, int s) { return s * pl.S - max(0, s - pl.nS); }
__device__ __forceinline__ int seg_rows(const SegPlan &pl, int s) { return pl.S - ((s < 0 ? pl.G - 1 : s) >= pl.nS); }

// The lane of a line that lies whole in this block's tile (line at base, rows
// P elements apart, pl.pad more after every full segment).
template <int SEG, bool FULL, typename E>
__device__ __forceinline__ SegLane<E> seg_lane(const SegPlan &pl, E *base, int seg, int N, int P) {
    SegLane<E> s;
    s.seg = seg;
    if constexpr (FULL) {
        s.k0 = 0;
        s.row = base + seg * (SEG * P + pl.pad);
        s.lo = seg > 0 ? s.row - pl.pad : base + N * P + (pl.G - 1) * pl.pad;
        s.hi = seg < pl.G - 1 ? s.row + SEG * P + pl.pad : base;
    } else {
        const int n0 = seg_row0(pl, seg), len = pl.S - (seg >= pl.nS);
        s.k0 = SEG - len;
        s.row = base + (n0 - s.k0) * P;
        s.lo = n0 > 0 ? s.row : s.row + N * P;
        s.hi = seg < pl.G - 1 ? base + (n0 + len) * P : base;
    }
    return s;
}

// The window of a segment: register row k at w[k + H], H rows either side.
// Rows before the segment's own (ragged segments) come from the halo or stay
// zero; the callers zero their right-hand sides.
template <int SEG, bool FULL, int H, typename W, typename E, typename I, typename LD>
__device__ __forceinline__ void seg_load(W (&w)[SEG + 2 * H], const SegLane<E> &s, I P, LD &&ld) {
#pragma unroll
    for (int k = -H; k < SEG; ++k) {
        if (FULL) {
            w[k + H] = k < 0 ? ld(s.lo + k * P) : ld(s.row + k * P);
        } else if (k < kSegSlack) {
            w[k + H] = W{};
            if (k >= s.k0 - H) w[k + H] = k < s.k0 ? ld(s.lo + k * P) : ld(s.row + k * P);
        } else {
            w[k + H] = ld(s.row + k * P);
        }
    }
#pragma unroll
    for (int h = 0; h < H; ++h) w[SEG + H + h] = ld(s.hi + h * P);
}

// Right-hand sides from a window (taps scaled by 1/h, 1/h^2 and 1 + l^2): the
// differences first, so that their products round relative to the differences.
template <int SEG, typename R>
__device__ __forceinline__ R seg_r1(const R (&w)[SEG + 4], const SegOp<R> &o, int k) {
    return fma(o.s[1], w[k + 3] - w[k + 1], o.s[2] * (w[k + 4] - w[k]));
}
template <int SEG, typename R>
__device__ __forceinline__ R seg_r2(const R (&w)[SEG + 4], const SegOp<R> &o, int k) {
    return fma(o.s[1], (w[k + 3] - w[k + 2]) - (w[k + 2] - w[k + 1]),
               o.s[2] * ((w[k + 4] - w[k + 2]) - (w[k + 2] - w[k])));
}
// 64 bits: the same by second differences D, s1 D_k + s2 (D_{k-1} + 2 D_k + D_{k+1}),
// o.s[0] = s1 + 2 s2.  Neighbouring rows share them, so that a row takes five
// operations, as many as the plain sum of taps and values, whose products round
// relative to the values (128 points: rms error 3e-16 of the result instead of 4e-15).
template <int SEG>
__device__ __forceinline__ double seg_r2(const double (&w)[SEG + 4], const SegOp<double> &o, int k) {
    const double da = w[k + 1] - w[k], db = w[k + 2] - w[k + 1], dc = w[k + 3] - w[k + 2], dd = w[k + 4] - w[k + 3];
    return fma(o.s[2], (db - da) + (dd - dc), o.s[0] * (dc - db));
}
template <int SEG, typename R>
__device__ __forceinline__ R seg_r3(const R (&w)[SEG + 8], const SegOp<R> &o, int k) {
    R r = o.s[0] * w[k + 4];
#pragma unroll
    for (int h = 1; h <= 4; ++h) r = fma(o.s[h], w[k + 4 - h] + w[k + 4 + h], r);
    return r;
}

// y: right-hand sides (zero in rows before k0).  Forward from zero: the
// segment's end value.
template <int SEG, typename R>
__device__ __forceinline__ R seg_fwd(R (&y)[SEG], const SegOp<R> &o) {
    R c = y[0];
#pragma unroll
    for (int k = 1; k < SEG; ++k) y[k] = c = fma(o.nl, c, y[k]);
    return c;
}
// Add the value entering the segment (KU: rows that take it), then backward
// from zero: the value at the segment's first row.
template <int SEG, bool FULL, int KU, typename R>
__device__ __forceinline__ R seg_bwd(R (&y)[SEG], const SegOp<R> &o, const SegPlan &pl, int k0, R in) {
    constexpr int KF = KU + (FULL ? 0 : kSegSlack) < SEG ? KU + (FULL ? 0 : kSegSlack) : SEG;
    if constexpr (!FULL) in *= k0 == pl.kS ? o.iS : o.iS1;  // the powers count from row k0
#pragma unroll
    for (int k = 0; k < KF; ++k) y[k] = fma(o.pw[k], in, y[k]);
    R c = y[SEG - 1], b = c;
#pragma unroll
    for (int k = SEG - 2; k >= 0; --k) {
        y[k] = c = fma(o.nl, c, y[k]);
        if (!FULL && k <= kSegSlack) b = k == k0 ? c : b;
    }
    return FULL ? c : b;
}
// Add the value at the next segment's first row.
template <int SEG, int KU, typename R>
__device__ __forceinline__ void seg_end(R (&y)[SEG], const SegOp<R> &o, R in) {
#pragma unroll
    for (int k = 0; k < (KU < SEG ? KU : SEG); ++k) y[SEG - 1 - k] = fma(o.pw[k], in, y[SEG - 1 - k]);
}

// Backward from zero without the entering value: the value at the first row.
template <int SEG, bool FULL, typename R>
__device__ __forceinline__ R seg_bwd0(R (&y)[SEG], const SegOp<R> &o, int k0) {
    R c = y[SEG - 1], b = c;
#pragma unroll
    for (int k = SEG - 2; k >= 0; --k) {
        y[k] = c = fma(o.nl, c, y[k]);
        if (!FULL && k <= kSegSlack) b = k == k0 ? c : b;
    }
    return FULL ? c : b;
}
// Both values added at once to a segment solved from zero on both sides, where
// they reach no further than the segment: `in` entered the forward pass (the
// backward pass answers (-l)^(k+1) with (-l)^(k+1) / (1 - l^2)), `next` is the
// solution's value after the last row.
template <int SEG, bool FULL, int KU, typename R>
__device__ __forceinline__ void seg_close(R (&y)[SEG], const SegOp<R> &o, const SegPlan &pl, int k0, R in, R next) {
    constexpr int KF = KU + (FULL ? 0 : kSegSlack) < SEG ? KU + (FULL ? 0 : kSegSlack) : SEG;
    in *= o.geo;
    if constexpr (!FULL) in *= k0 == pl.kS ? o.iS : o.iS1;  // the powers count from row k0
#pragma unroll
    for (int k = 0; k < KF; ++k) y[k] = fma(o.pw[k], in, y[k]);
    seg_end<SEG, KU>(y, o, next);
}

// What enters this lane's segment: e of the DIR-side neighbours (DIR = -1:
// segments before, +1: after), weighted.  lane0: the line's first lane, its
// segments 2^lgst lanes apart.
template <int DIR, typename R>
__device__ __forceinline__ R seg_carry(R e, const SegOp<R> &o, const SegPlan &pl, int seg, int lane0, int lgst) {
    R c = R(0);
    for (int t = o.T; t >= 1; --t) {
        const int src = (seg + DIR * t) & (pl.G - 1);
        const R es = __shfl_sync(0xffffffffu, e, lane0 + (src << lgst));
        c = fma(src < pl.nS ? o.qS : o.qS1, c, es);
    }
    return c * o.wrap;
}

// The whole solve, all segments of the line in this warp.
template <int SEG, bool FULL, int KU, typename R>
__device__ __forceinline__ void seg_solve(R (&y)[SEG], const SegOp<R> &o, const SegPlan &pl, int seg, int k0,
                                          int lane0, int lgst) {
    const R e = seg_fwd<SEG>(y, o);
    const R b = seg_bwd<SEG, FULL, KU>(y, o, pl, k0, seg_carry<-1>(e, o, pl, seg, lane0, lgst));
    seg_end<SEG, KU>(y, o, seg_carry<1>(b, o, pl, seg, lane0, lgst));
}

// Store the segment's own rows.
template <int SEG, bool FULL, typename E, typename I, typename ST>
__device__ __forceinline__ void seg_store(const SegLane<E> &s, I P, ST &&st) {
#pragma unroll
    for (int k = 0; k < SEG; ++k)
        if (FULL || k >= kSegSlack || k >= s.k0) st(s.row + k * P, k);
}

// The right-hand sides of two solves of the pair-interleaved tile (element n
// of a pair: a float2).  MODE 0: lane x's field by the 1st (y1) and 2nd (y2)
// derivative, 1: both lanes' fields by the 1st derivative, 2: lane x's field
// alone by the 1st, 3: lane x's field by the 1st, lane y's by the 2nd.
template <int SEG, bool FULL, int MODE>
__device__ __forceinline__ void seg_pair_rhs(float (&y1)[SEG], float (&y2)[SEG], const SegLane<float2> &s, int P,
                                             const SegOp<float> &o1, const SegOp<float> &o2) {
    float w1[SEG + 4], w2[SEG + 4];
    if constexpr (MODE == 0 || MODE == 2) {
        seg_load<SEG, FULL, 2>(w1, s, P, [](const float2 *p) { return p->x; });
    } else {
        float2 w[SEG + 4];
        seg_load<SEG, FULL, 2>(w, s, P, [](const float2 *p) { return *p; });
#pragma unroll
        for (int k = 0; k < SEG + 4; ++k) { w1[k] = w[k].x; w2[k] = w[k].y; }
    }
#pragma unroll
    for (int k = 0; k < SEG; ++k) {
        y1[k] = seg_r1<SEG>(w1, o1, k);
        if constexpr (MODE == 0) y2[k] = seg_r2<SEG>(w1, o2, k);
        if constexpr (MODE == 1) y2[k] = seg_r1<SEG>(w2, o1, k);
        if constexpr (MODE == 3) y2[k] = seg_r2<SEG>(w2, o2, k);
        if constexpr (MODE == 2) y2[k] = 0.f;
        if (!FULL && k < kSegSlack && k < s.k0) y1[k] = y2[k] = 0.f;
    }
}

// Two solves of the tile in place, all segments of their lines in this warp.
template <int SEG, bool FULL, int MODE>
__device__ __forceinline__ void seg_pair(const SegLane<float2> &s, int P, const SegOp<float> &o1, const SegOp<float> &o2,
                                         const SegPlan &pl, int lane0, bool active) {
    float y1[SEG], y2[SEG];
    seg_pair_rhs<SEG, FULL, MODE>(y1, y2, s, P, o1, o2);
    seg_solve<SEG, FULL, kSegRows1>(y1, o1, pl, s.seg, s.k0, lane0, pl.lgLW);
    if constexpr (MODE == 0 || MODE == 3) seg_solve<SEG, FULL, kSegRows2>(y2, o2, pl, s.seg, s.k0, lane0, pl.lgLW);
    if constexpr (MODE == 1) seg_solve<SEG, FULL, kSegRows1>(y2, o1, pl, s.seg, s.k0, lane0, pl.lgLW);
    __syncwarp();  // every lane of the line has read its window
    if (!active) return;
    seg_store<SEG, FULL>(s, P, [&](float2 *p, int k) {
        if constexpr (MODE == 2) p->x = y1[k];
        else *p = make_float2(y1[k], y2[k]);
    });
}

// One solve of a planar tile: the KIND-th derivative of the segment at `s`,
// its rows stored to the same places `shift` elements on (0: in place).
template <int SEG, bool FULL, int KIND, typename R>
__device__ __forceinline__ void seg_one(const SegLane<R> &s, int P, const SegOp<R> &o, const SegPlan &pl, int lane0,
                                        bool active, int shift) {
    R y[SEG];
    {
        R w[SEG + 4];
        seg_load<SEG, FULL, 2>(w, s, P, [](const R *p) { return *p; });
#pragma unroll
        for (int k = 0; k < SEG; ++k) {
            y[k] = KIND == 1 ? seg_r1<SEG>(w, o, k) : seg_r2<SEG>(w, o, k);
            if (!FULL && k < kSegSlack && k < s.k0) y[k] = R(0);
        }
    }
    constexpr int K1 = sizeof(R) == 4 ? kSegRows1 : kSegRowsAll, K2 = sizeof(R) == 4 ? kSegRows2 : 24;
    seg_solve<SEG, FULL, KIND == 1 ? K1 : K2>(y, o, pl, s.seg, s.k0, lane0, pl.lgLW);
    __syncwarp();  // every lane of the line has read its window
    if (active) seg_store<SEG, FULL>(s, P, [&](R *p, int k) { p[shift] = y[k]; });
    __syncwarp();
}

// The filter (nine symmetric taps) of the segment at `s` in place.  FP32: o is
// the correction F - I, added to the value (ADD); FP64: o is F itself.
template <int SEG, bool FULL, bool ADD, typename R>
__device__ __forceinline__ void seg_filter(const SegLane<R> &s, int P, const SegOp<R> &o, const SegPlan &pl,
                                           int lane0, bool active) {
    R y[SEG];
    {
        R w[SEG + 8];
        seg_load<SEG, FULL, 4>(w, s, P, [](const R *p) { return *p; });
#pragma unroll
        for (int k = 0; k < SEG; ++k) {
            y[k] = seg_r3<SEG>(w, o, k);
            if (!FULL && k < kSegSlack && k < s.k0) y[k] = R(0);
        }
    }
    seg_solve<SEG, FULL, kSegRowsAll>(y, o, pl, s.seg, s.k0, lane0, pl.lgLW);
    __syncwarp();  // every lane of the line has read its window
    if (active) seg_store<SEG, FULL>(s, P, [&](R *p, int k) { *p = ADD ? *p + y[k] : y[k]; });
}

// ---------------------------------------------------------------------
// lines split over a thread-block cluster
// ---------------------------------------------------------------------
// A tile of 32 neighbouring lines is 128 bytes a row, whole memory lines; 16
// solves of 32 lines fit one SM's shared memory for 64 rows only, so a cluster
// of C blocks holds the line, B = one or two 32-row segments a block.  One (up to
// 256 points) leaves room for two blocks an SM, one solving while the other's
// loads and stores run.  Halo rows are read from the neighbours' shared memory;
// the carries (T = 1: the plan keeps segments long enough for the nearest
// neighbour alone) cross in one exchange: every segment is solved from zero on
// both sides, its last forward value goes to the next block's mailbox and its
// first solution value to the previous one's (seg_close).
// Why: beyond the L2 the memory system delivers in proportion to the bytes a
// tile's row takes of its 128-byte line -- a copy kernel of z tiles on 256^3
// measured 2.0 / 3.9 / 6.5 TB/s at 8 / 16 / 32 FP32 lines a row (5.2 / 5.6 /
// 5.3 TB/s at 128^3, which the L2 holds).  The 8-line tiles that whole lines
// leave room for at N = 256: z 6.66 ms a step; clusters of 4 with two segments a block
// 4.03, of 8 with one 3.20.
constexpr int kClLines = 32;  // (kClusterLines)

__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of p (this block's shared memory) in block `rank` of the cluster.
template <typename E>
__device__ __forceinline__ E *cluster_map(E *p, int rank) {
    E *r;
    asm("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(p), "r"(rank));
    return r;
}

// Lines between walls: the first and last two rows' stencils are one-sided and
// the factors converge to the periodic ones within 20 rows of the ends (they
// approach like l^2n), so the first and last segment of a line take their
// factors from tables (32 register rows each, the same for all lanes) and the
// others run as on a periodic line, as does every exchange.
struct WallOp {
    float bt[4][6];         // the explicit rows (scaled as the taps): 0, 1 from row 0 on, N-2, N-1 from row N-6 on
    float s[2][32], f[2][32], b[2][32];  // y_n = s_n r_n + f_n y_{n-1}, x_n = y_n + b_n x_{n+1}
};

// One solve of the first (END = 0) or last segment from zero: its last forward
// value into e, its first solution value into b.  x: the segment's first row,
// in the tile (of one lane of the pair).  END and the rows are
// known to the compiler, so that a table's entry is an operand of its operation
// and not a load (y of 256x128x42, 64 of 128 rows in such segments: 49.3 us a
// stage with tables in memory, 44.8 so).
template <int SEG, bool FULL, int END>
__device__ __forceinline__ void wall_solve(float (&y)[SEG], const float *x, int P2, const WallOp &w, int k0, float &e,
                                           float &b) {
    // the explicit rows.  (Their coefficients sum to zero: differences from the
    // wall value, so that rounded coefficients make no derivative of a constant.)
    const float *p = x + (END ? SEG - 6 : FULL ? 0 : k0) * P2;
    const float v0 = p[END ? 5 * P2 : 0];
    float r0 = 0.f, r1 = 0.f;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const float v = p[j * P2] - v0;
        r0 = fmaf(w.bt[2 * END][j], v, r0);
        r1 = fmaf(w.bt[2 * END + 1][j], v, r1);
    }
    if (END) {
        y[SEG - 2] = r0;
        y[SEG - 1] = r1;
    } else if (FULL) {
        y[0] = r0;
        y[1] = r1;
    } else {
        // (selects: as an assignment to row k0 the array leaves the registers:
        // y of 128x127x128 101 us a stage, 73 so)
#pragma unroll
        for (int k = 0; k < kSegSlack + 2; ++k) y[k] = k == k0 ? r0 : k == k0 + 1 ? r1 : y[k];
    }
    float c = 0.f;
#pragma unroll
    for (int k = 0; k < SEG; ++k) y[k] = c = fmaf(w.f[END][k], c, w.s[END][k] * y[k]);
    e = c;
    c = b = 0.f;
#pragma unroll
    for (int k = SEG - 1; k >= 0; --k) {
        y[k] = c = fmaf(w.b[END][k], c, y[k]);
        if (!FULL && k <= kSegSlack) b = k == k0 ? c : b;
    }
    if (FULL) b = c;
}
// A task's two solves there: y1 by w1, y2 by w2 (dd: a second derivative, of the
// lane x field unless MIX) or w1.
template <int SEG, bool FULL, bool MIX, int END>
__device__ __forceinline__ void wall_task(float (&y1)[SEG], float (&y2)[SEG], const float *x, int P2, const WallOp &w1,
                                          const WallOp &w2, int k0, bool dd, bool single, float2 &e, float2 &b) {
    wall_solve<SEG, FULL, END>(y1, x, P2, w1, k0, e.x, b.x);
    if (dd) wall_solve<SEG, FULL, END>(y2, MIX ? x + 1 : x, P2, w2, k0, e.y, b.y);
    else if (!single) wall_solve<SEG, FULL, END>(y2, x + 1, P2, w1, k0, e.y, b.y);
    else e.y = b.y = 0.f;
}

// The solves of a sweep tile (tasks as run_seg_tasks), one unit a warp: pl.B
// segments of 32 / pl.B lines of one task.  MIX: tasks 0..3 take the second
// derivative of the lane y field.  mail: 2 * 8 * kClLines float2s.  Every
// thread of every block of the cluster calls it.
// WALL: w1, w2 (one segment a block).
template <bool FULL, int NT, bool SINGLE, bool MIX = false, bool WALL = false>
__device__ __forceinline__ void run_cluster_tasks(float2 *tile, int pstride2, float2 *mail, const SegPlan &pl,
                                                  const SegOp<float> &o1, const SegOp<float> &o2, int rank, int tid,
                                                  const WallOp *w1 = nullptr, const WallOp *w2 = nullptr) {
    constexpr int SEG = 32, P = kClLines;
    const int B = pl.B, warp = tid >> 5, t = B == 2 ? warp >> 1 : warp, half = B == 2 ? (tid >> 4) & 1 : 0;
    const int l = B == 2 ? ((warp & 1) << 4) | (tid & 15) : tid & 31;
    const int C = pl.C, prev = rank > 0 ? rank - 1 : C - 1, next = rank < C - 1 ? rank + 1 : 0;
    const int seg = B * rank + half;
    const bool first = half == 0, last = half == B - 1;  // of this block
    float2 *line = tile + t * pstride2 + l;
    SegLane<float2> s;
    s.seg = seg;
    const int n0 = seg_row0(pl, seg) - seg_row0(pl, B * rank), len = pl.S - (seg >= pl.nS);
    s.k0 = FULL ? 0 : SEG - len;
    s.row = line + (n0 - s.k0) * P;
    // (rows of the previous block: its last row precedes this block's first)
    const int nprev = FULL ? SEG * B : seg_row0(pl, B * (prev + 1)) - seg_row0(pl, B * prev);
    s.lo = first ? cluster_map(line + (nprev - s.k0) * P, prev) : cluster_map(s.row, rank);
    s.hi = last ? cluster_map(line, next) : cluster_map(line + (n0 + len) * P, rank);
    const bool dd = t < 4, single = SINGLE && t == NT - 1;
    const SegOp<float> &ob = dd ? o2 : o1;
    float y1[SEG], y2[SEG];
    if (dd) seg_pair_rhs<SEG, FULL, MIX ? 3 : 0>(y1, y2, s, P, o1, o2);
    else if (single) seg_pair_rhs<SEG, FULL, 2>(y1, y2, s, P, o1, o2);
    else seg_pair_rhs<SEG, FULL, 1>(y1, y2, s, P, o1, o2);
    float2 e, b;  // the segment's last forward value, its first solution value
    if (WALL && (rank == 0 || rank == C - 1)) {
        const float *x = reinterpret_cast<const float *>(s.row);
        if (rank == 0) wall_task<SEG, FULL, MIX, 0>(y1, y2, x, 2 * P, *w1, *w2, s.k0, dd, single, e, b);
        else wall_task<SEG, FULL, MIX, 1>(y1, y2, x, 2 * P, *w1, *w2, s.k0, dd, single, e, b);
    } else {
        e.x = seg_fwd<SEG>(y1, o1);
        b.x = seg_bwd0<SEG, FULL>(y1, o1, s.k0);
        e.y = b.y = 0.f;
        if (!single) {
            e.y = seg_fwd<SEG>(y2, ob);
            b.y = seg_bwd0<SEG, FULL>(y2, ob, s.k0);
        }
    }
    float2 *box = mail + t * kClLines + l, *box2 = box + 8 * kClLines;
    if (last) *cluster_map(box, next) = e;
    if (first) *cluster_map(box2, prev) = b;
    float2 in, nb;  // the other half's, where this block holds two segments
    in.x = __shfl_sync(0xffffffffu, e.x, tid & 15);
    in.y = __shfl_sync(0xffffffffu, e.y, tid & 15);
    nb.x = __shfl_sync(0xffffffffu, b.x, (tid & 15) | 16);
    nb.y = __shfl_sync(0xffffffffu, b.y, (tid & 15) | 16);
    // the neighbours' values are there, and every window has been read (the
    // last access to another block's shared memory)
    cluster_sync();
    if (first) in = *box;
    if (last) nb = *box2;
    // the next segment's first value answers this one's forward value too
    nb.x = fmaf(e.x, o1.nl * o1.geo, nb.x);
    nb.y = fmaf(e.y, ob.nl * ob.geo, nb.y);
    if (WALL && rank == 0) in = make_float2(0.f, 0.f);
    if (WALL && rank == C - 1) nb = make_float2(0.f, 0.f);
    seg_close<SEG, FULL, kSegRows1>(y1, o1, pl, s.k0, in.x, nb.x);
    if (dd) seg_close<SEG, FULL, kSegRows2>(y2, o2, pl, s.k0, in.y, nb.y);
    else if (!single) seg_close<SEG, FULL, kSegRows1>(y2, o1, pl, s.k0, in.y, nb.y);
    seg_store<SEG, FULL>(s, P, [&](float2 *p, int k) { *p = make_float2(y1[k], y2[k]); });
}

// ---------------------------------------------------------------------
// FP64 lines, one thread a line
// ---------------------------------------------------------------------
// The plain form is bound by FP64 issue (two operations an SM and clock), so
// its solves take the fewest operations: one thread walks the R rows of its
// line that this block holds, in place in shared memory (4 or 5 operations for
// the stencil, one a row forward, one backward), and the carries touch only
// the K rows that they reach: 6.6 (first derivative) and 7.4 operations a row
// at R = 128 against 9 of the Thomas sweep with its Sherman-Morrison
// correction.  The line's other rows are in the blocks of a cluster, as in
// run_cluster_tasks; R >= 40 there, so that a carry crosses one block at most.
// Whole lines of one block: the circle closes on itself (wrap).
constexpr int kSeqRows = 44;  // powers kept: 0.382^41 < 2^-56
struct SeqOp {
    double nl, s0, s1, s2, wrap;
    int K;
    double pw[kSeqRows];  // (-l)^(k+1), k < K (among the kernel's arguments: a
                          // first read from memory costs a short line's solve
                          // as much as its arithmetic)
};

// The two rows before a segment's first and the two after its last, read
// before any row is written.
struct SeqHalo {
    double lo[2], hi[2];
};
__device__ __forceinline__ SeqHalo seq_halo(const double *lo, const double *hi, int P) {
    return {{lo[-2 * P], lo[-P]}, {hi[0], hi[P]}};
}
// KIND 1, 2.  Returns the end value.
template <int KIND>
__device__ __forceinline__ double seq_fwd(double *d, int P, int R, const SeqOp &o, const SeqHalo &h) {
    double w0 = h.lo[0], w1 = h.lo[1], w2 = d[0], w3 = d[P];
    const double nl = o.nl, s0 = o.s0, s1 = o.s1, s2 = o.s2;
    double y = 0.0;
    auto row = [&](double w4) {
        const double r = KIND == 1 ? fma(s1, w3 - w1, s2 * (w4 - w0)) : fma(s2, w4 + w0, fma(s1, w3 + w1, s0 * w2));
        y = fma(nl, y, r);
        w0 = w1; w1 = w2; w2 = w3; w3 = w4;
    };
    double *q = d;
    int n = 0;
    for (; n + 6 <= R; n += 4, q += 4 * P) {
        double c[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = q[(j + 2) * P];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            row(c[j]);
            q[j * P] = y;
        }
    }
    for (; n < R; ++n, q += P) {
        row(n + 2 < R ? q[2 * P] : n + 2 == R ? h.hi[0] : h.hi[1]);
        q[0] = y;
    }
    return y;
}
// Backward, `in` entering at the first row; returns the first row's value.
__device__ __forceinline__ double seq_bwd(double *d, int P, int R, const SeqOp &o, double in) {
    const double nl = o.nl;
    const int K = min(o.K, R);
    double x = 0.0;
    double *q = d + (R - 1) * P;
    int n = R;
    for (; n - 4 >= K; n -= 4, q -= 4 * P) {
        double c[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = q[-j * P];
#pragma unroll
        for (int j = 0; j < 4; ++j) q[-j * P] = x = fma(nl, x, c[j]);
    }
    for (; n > K; --n, q -= P) q[0] = x = fma(nl, x, q[0]);
    for (; n - 4 >= 0; n -= 4, q -= 4 * P) {
        double c[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = fma(o.pw[n - 1 - j], in, q[-j * P]);
#pragma unroll
        for (int j = 0; j < 4; ++j) q[-j * P] = x = fma(nl, x, c[j]);
    }
    for (; n > 0; --n, q -= P) q[0] = x = fma(nl, x, fma(o.pw[n - 1], in, q[0]));
    return x;
}
__device__ __forceinline__ void seq_end(double *d, int P, int R, const SeqOp &o, double in) {
    const int K = min(o.K, R);
    double *q = d + (R - 1) * P;
#pragma unroll 4
    for (int k = 0; k < K; ++k) q[-k * P] = fma(o.pw[k], in, q[-k * P]);
}

// The solves of a tile of L lines (a power of two <= 32), planar buffers
// `stride` apart: n1 first derivatives in buffers 0 .., then second derivatives
// of the first four fields in n1 .. n1 + 3, each in place.  A line's segments:
// one a block of a cluster of pl.C blocks (R rows here), or pl.G in this block
// (R: all rows).  Warps are uniform: the second derivatives start at a warp's
// first lane.  mail: 2 (n1 + 4) L doubles per segment of the block.  Every
// thread of every block of the cluster calls it.
__device__ __forceinline__ void run_seq_tasks(double *tile, int stride, double *mail, int n1, int L, int lgL, int R,
                                              const SegPlan &pl, const SeqOp &o1, const SeqOp &o2, int rank, int tid) {
    const int C = pl.C, B = C > 1 ? 1 : pl.G;      // segments of a line in this block: 1, 2 or 4
    const int per = 32 >> lgL;                     // solves a warp holds
    const int n1p = (n1 * B + per - 1) & ~(per - 1);
    int k = tid >> lgL;
    const int l = tid & (L - 1);
    const bool second = k >= n1p;
    const bool on = second ? k < n1p + 4 * B : k < n1 * B;
    if (second) k -= n1p;
    if (!on) k = 0;
    const int h = k & (B - 1);
    k = (B == 4 ? k >> 2 : B == 2 ? k >> 1 : k) + (second && on ? n1 : 0);
    double *line = tile + k * stride + l, *d = line + (B > 1 ? seg_row0(pl, h) : 0) * L;
    const int rows = B > 1 ? seg_rows(pl, h) : R;
    double *mbox = mail + B * k * L + l, *box = mbox + h * L, *box2 = box + B * (n1 + 4) * L;
    const SeqOp &o = second ? o2 : o1;
    double v = 0.0;
    if (C > 1) {
        const int prev = rank > 0 ? rank - 1 : C - 1, next = rank < C - 1 ? rank + 1 : 0;
        const double *lo = cluster_map(d + seg_rows(pl, rank - 1) * L, prev), *hi = cluster_map(d, next);
        const SeqHalo halo = seq_halo(lo, hi, L);
        cluster_sync();
        // (idle lanes have the first line's addresses, whose rows are being written now)
        if (on) v = second ? seq_fwd<2>(d, L, R, o, halo) : seq_fwd<1>(d, L, R, o, halo);
        if (on) *cluster_map(box, next) = v;
        cluster_sync();
        if (on) {
            v = seq_bwd(d, L, R, o, *box);
            *cluster_map(box2, prev) = v;
        }
        cluster_sync();  // (the last access to another block's shared memory)
        if (on) seq_end(d, L, R, o, *box2);
    } else if (B > 1) {
        const int hp = (h - 1) & (B - 1), hn = (h + 1) & (B - 1);
        const double *lo = h ? d : line + R * L, *hi = hn ? d + rows * L : line;
        const SeqHalo halo = seq_halo(lo, hi, L);
        __syncthreads();
        // (idle lanes have the first line's addresses, whose rows are being written now)
        if (on) v = second ? seq_fwd<2>(d, L, rows, o, halo) : seq_fwd<1>(d, L, rows, o, halo);
        if (on) mbox[hn * L] = v;
        __syncthreads();
        if (on) {
            v = seq_bwd(d, L, rows, o, *box);
            mbox[hp * L + B * (n1 + 4) * L] = v;
        }
        __syncthreads();
        if (on) seq_end(d, L, rows, o, *box2);
    } else if (on) {
        const SeqHalo halo = seq_halo(d + R * L, d, L);
        if (second) v = seq_fwd<2>(d, L, R, o, halo);
        else v = seq_fwd<1>(d, L, R, o, halo);
        v = seq_bwd(d, L, R, o, v * o.wrap);
        seq_end(d, L, R, o, v * o.wrap);
    }
}

}  // namespace cs3d
