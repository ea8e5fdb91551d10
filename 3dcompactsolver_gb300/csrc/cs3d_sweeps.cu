// cs3d_sweeps.cu -- the directional sweep kernels of one RK stage, the
// compact filter and the single-operator kernel (sm_103a).
//
// One stage is three fused directional sweeps.  A block takes a tile of lines
// along the sweep direction -- whole lines, or 32 lines' rows of one block of a
// cluster -- and runs three phases:
//
//   A  load the tile's inputs (batched, several points per thread in
//      flight), form primitives and fluxes, stage every line-solve input in
//      shared memory ([position][line] layout);
//   B  solve.  A task is two line solves run together -- the 1st and 2nd
//      derivative of one field, or the 1st derivative of two.  Mixed form:
//      segments of 16 to 32 rows in registers (run_seg_x, run_cluster_tasks);
//      plain form: one thread walks its block's rows (run_seq_tasks); Thomas
//      sweeps with precomputed factors for the lines that neither cuts (FP64
//      wall lines; mixed ones along x, below 40 or above 256 points, or where
//      mixed_plan says so; mixed periodic ones of 8 or above 512 points);
//   C  consume the derivatives point by point.
//
//   sweep x : primitives, Euler x-fluxes, 13 x-solves; writes Ux,Vx,Wx,Tx,
//             the plain form's p, mu, mu'(T) and the linear x-part of the
//             five right-hand sides
//   sweep y : 15 y-solves (incl. the cross derivatives Uxy, Vxy); writes
//             Uy,Vy,Wy,Ty and adds the linear y-part
//   sweep z : 16 z-solves (incl. d/dz of Ux+Vy, Wx, Wy), the nonlinear viscous
//             terms, dt, the wall/sponge increment fix-up and the RK4 /
//             TVD-RK3 update of the conserved state (k_sponge_source, where
//             there is a sponge, runs before it)
//
// The reference instead stores ~48 derivative fields and makes ~54 layout
// transposes per stage (CSolver_AWS.cpp:829-1243).  Lines along y and z are
// read in place in the XYZ layout: a tile is L consecutive x-columns, so every
// global access is a contiguous row segment; x-lines are transposed into
// shared memory on load.
//
// T is the work precision: double for the plain form, float for the mixed
// form.  The conserved state (q1, q2, and qk where kept) is FP64.
#include <cstdio>
#include <cmath>
#include "cs3d_tile.cuh"

namespace cs3d {

// Points per thread in flight in the point loops of the mixed form (measured
// at 128^3 and 256^3; deeper batches spill or run no faster).  The x sweep and
// every load phase: 4; the z update: 1 (its 33 loads a point are enough).
constexpr int kFilterBatch = 4;         // the mixed filter's load and store loops
constexpr int kFilterConsumeBatch = 2;  // the mixed filter's consume loop
constexpr int kYConsumeBatch = 4;       // the y sweep's consume phase
// Resident blocks per SM the mixed-form kernels are compiled for: the x sweep 3
// blocks of 256 threads (80 registers; ragged segments 2), y and z 512 threads
// (128 registers: two cluster blocks of 256), the Thomas filter 4 (64).
constexpr int kFilterMinBlocks = 4;
constexpr int kMinBlocksX = 3, kMinBlocksY = 1, kMinBlocksZ = 1;

// Mixed form: the y and z sweeps form the pressure from what they read anyway
// and the viscosity and its slope from T (a hardware log2 and exp2), so that x
// stores neither: 32 of about 380 bytes a point and stage.  The plain form,
// bound by FP64 issue, stores them.
template <typename T>
constexpr bool kRecompute = sizeof(T) == 4;

// The sweep kernels take the shared-memory pitch of their tile as a template
// parameter PC (0: read at run time).  The launcher instantiates the mixed
// form's usual pitches (x: 9 and 5; y, z: 16 and 8), where every
// shared-memory access of a solve chunk becomes an immediate off one base
// register: x 0.358 -> 0.336 ms, y and z 2-4% faster per step at 128^3.
//
// SEG > 0: the segmented solves of cs3d_seg.cuh, SEG rows a segment (kSeq: the
// plain form's sequential ones), FULL when the line length is a multiple; CL: the
// line over a cluster; WALL: between walls.  The tile then has no line factors
// and its solutions need no correction on read.  SEG = 0: the Thomas solves with
// precomputed factors (FP64 wall lines, and lengths that no plan cuts).
template <typename T, int SEG>
struct TileOf {
    using SM = typename SweepSmem<T>::type;
    static __device__ __forceinline__ SM at(int nbuf, int L, int P, int N, const SegPlan &) {
        return SweepSmem<T>::at(smem_raw, nbuf, L, P, N);
    }
    static __device__ __forceinline__ void put1f(const SM &sm, int t, int o, T v) { put1(sm, t, o, v); }
    static __device__ __forceinline__ Zn<T> z(const LineOp<T> &d1, const LineOp<T> &d2, int n) { return zn(d1, d2, n); }
    static __device__ __forceinline__ void two(const SM &sm, int t, const Pt &p, int L, T za, T zb, T &a, T &b) {
        get2(sm, t, p, L, za, zb, a, b);
    }
    static __device__ __forceinline__ T one(const SM &sm, int k, const Pt &p, int L, T z) { return get1(sm, k, p, L, z); }
};
// FP64, periodic lines: planar buffers of the sequential solves, the n1 first
// derivatives, then the four second derivatives (each solved in place, so the
// load phase stores those fields twice).
constexpr int kSeq = kSeqSeg;
struct SmemSeq {
    double *buf;
    int stride, n1;
    __device__ double &at(int k, int o) const { return buf[k * stride + o]; }
};
template <>
struct TileOf<double, kSeq> {
    using SM = SmemSeq;
    static __device__ __forceinline__ SM at(int n1, int L, int, int R, const SegPlan &) {
        return {reinterpret_cast<double *>(smem_raw), seq_stride(R, L), n1};
    }
    static __device__ __forceinline__ void put1f(const SM &sm, int t, int o, double v) {
        if (t < 4) {
            sm.at(t, o) = v;
            sm.at(sm.n1 + t, o) = v;
        } else {
            sm.at(2 * t - 4, o) = v;
        }
    }
    static __device__ __forceinline__ Zn<double> z(const LineOp<double> &, const LineOp<double> &, int) { return {0.0, 0.0}; }
    static __device__ __forceinline__ void two(const SM &sm, int t, const Pt &p, int, double, double, double &a, double &b) {
        a = sm.at(t < 4 ? t : 2 * t - 4, p.o);
        b = sm.at(t < 4 ? sm.n1 + t : 2 * t - 3, p.o);
    }
    static __device__ __forceinline__ double one(const SM &sm, int, const Pt &p, int, double) { return sm.at(sm.n1 - 1, p.o); }
    static __device__ __forceinline__ double *mail(const SM &sm) { return sm.buf + (sm.n1 + 4) * sm.stride; }
};
__device__ __forceinline__ void put2(const SmemSeq &sm, int t, int o, double v0, double v1) {
    sm.at(2 * t - 4, o) = v0;
    sm.at(2 * t - 3, o) = v1;
}
// first derivatives of a sweep
constexpr int kSeqN1X = 9, kSeqN1Y = 11, kSeqN1Z = 12;
template <int SEG>
struct TileSegX {
    using SM = SmemSegX;
    static __device__ __forceinline__ SM at(int, int, int P, int N, const SegPlan &pl) {
        return {reinterpret_cast<float *>(smem_raw), seg_stride(N, P, pl.G, pl.pad)};
    }
    static __device__ __forceinline__ void put1f(const SM &sm, int t, int o, float v) { sm.at(2 * t, o) = v; }
    static __device__ __forceinline__ Zn<float> z(const LineOp<float> &, const LineOp<float> &, int) { return {0.f, 0.f}; }
    static __device__ __forceinline__ void two(const SM &sm, int t, const Pt &p, int, float, float, float &a, float &b) {
        a = sm.at(2 * t, p.o);
        b = sm.at(2 * t + 1, p.o);
    }
    static __device__ __forceinline__ float one(const SM &sm, int k, const Pt &p, int, float) { return sm.at(k, p.o); }
};
template <int SEG>
struct TileSeg {
    using SM = SmemPair;
    static __device__ __forceinline__ SM at(int, int, int P, int N, const SegPlan &pl) { return smem_pair_seg(P, N, pl); }
    static __device__ __forceinline__ void put1f(const SM &sm, int t, int o, float v) { sm.at(2 * t, o) = v; }
    static __device__ __forceinline__ Zn<float> z(const LineOp<float> &, const LineOp<float> &, int) { return {0.f, 0.f}; }
    static __device__ __forceinline__ void two(const SM &sm, int t, const Pt &p, int, float, float, float &a, float &b) {
        const float2 v = sm.pair(t)[p.o];
        a = v.x;
        b = v.y;
    }
    static __device__ __forceinline__ float one(const SM &sm, int k, const Pt &p, int, float) { return sm.at(k, p.o); }
};
template <> struct TileOf<float, 16> : TileSeg<16> {};
template <> struct TileOf<float, 24> : TileSeg<24> {};
template <> struct TileOf<float, 32> : TileSeg<32> {};

// ---------------------------------------------------------------------
// sweep x
// ---------------------------------------------------------------------
// Sweep task t solves into buffers 2t and 2t+1.  The FP32-mixed form's pair
// layout gives the last task of the x and y sweeps (one field) a spare second
// lane (XDUM, YDUM), which no thread solves; the FP64 form solves that field
// twice over in its own buffer.
enum { XU = 0, XU2, XV, XV2, XW, XW2, XT, XT2, XRU, XF1, XF2, XF3, XF4, XDUM, XNB2 };
constexpr int XNB = XDUM;
__constant__ Task kTasksX[7] = {{XU, XU, 0, XU, XU2, 1}, {XV, XV, 0, XV, XV2, 1}, {XW, XW, 0, XW, XW2, 1},
                                {XT, XT, 0, XT, XT2, 1}, {XRU, XRU, 0, XF1, XF1, 0},
                                {XF2, XF2, 0, XF3, XF3, 0}, {XF4, XF4, 0, XF4, XF4, 0}};
__constant__ Task kTasksX2[7] = {{XU, XU, 0, XU, XU2, 1}, {XV, XV, 0, XV, XV2, 1}, {XW, XW, 0, XW, XW2, 1},
                                 {XT, XT, 0, XT, XT2, 1}, {XRU, XRU, 0, XF1, XF1, 0},
                                 {XF2, XF2, 0, XF3, XF3, 0}, {XF4, XF4, 0, XF4, XDUM, 0}};

// FP64 segmented: 256 threads (128 registers), the 13 solves' segments of a tile
// fill 7 of 8 warps.  As 4-line tiles of 128 threads, 3 blocks an SM (3 of 4
// warps, a quarter of the lanes idle): 128^3 2.62 -> 2.52 ms a step.
template <typename T, int PC, int SEG = 0, bool FULL = false, int PLAIN = 0>
__global__ void __launch_bounds__(SEG == kSeq ? kSeqTpbX : sweep_threads<T>(0),
                                  sizeof(T) == 4 && (SEG == 0 || FULL) ? kMinBlocksX : 2) k_sweep_x(SweepArgs<T> a) {
    using TS = std::conditional_t<(SEG > 0 && sizeof(T) == 4), TileSegX<SEG>, TileOf<T, SEG>>;
    const int L = a.L, P = PC > 0 ? PC : a.P;
    const Tile t = make_tile<0>(a.g, L);
    const int N = t.N, NL = N * L, pad = FULL ? a.seg.pad : 0;
    const auto sm = TS::at(SEG == kSeq ? kSeqN1X : sizeof(T) == 4 ? XNB2 : XNB, L, P, N, a.seg);
    const GasParams gp = a.gas;
    // FP64 tiles: points across the lines first, pitch P = L (no pad column)
    constexpr bool kXLineFirst = sizeof(T) == 8;
    // phase A: primitives and the inputs of the x-solves
    struct InA { Pt pt; T q[5]; };
    batched<InA, sizeof(T) == 4 ? 4 : 2>(NL,
        [&](InA &in, int p) {
            in.pt = point<0, kXLineFirst>(t, p, L, P, a.lgL, a.divN, pad);
#pragma unroll
            for (int f = 0; f < 5; ++f) in.q[f] = a.qs[f][in.pt.gi];
        },
        [&](InA &in) {
            if (!in.pt.ok) return;
            const unsigned gi = in.pt.gi;
            PrimW<T> s = prim_w<T>(gp, in.q[0], in.q[1], in.q[2], in.q[3], in.q[4]);
            a.prim[0][gi] = s.U; a.prim[1][gi] = s.V; a.prim[2][gi] = s.W;
            a.prim[4][gi] = s.Tt;
            if constexpr (!kRecompute<T>) a.prim[3][gi] = s.p;
            // stage-start primitives: on stage 1, points of SPONGE faces (not
            // on a wall) use the state before the previous step's sponge
            // overwrite, which the reference's U,V,W,p,T arrays still hold.
            PrimW<T> ss = s;
            if (!PLAIN && a.use_backup) {
                int i, j, k;
                coords<0>(t, in.pt.l, in.pt.n, i, j, k);
                const int f = faces_of(a.g, i, j, k);
                if ((f & a.sponge_kind_faces) && !(f & a.wall_faces))
                    ss = prim_w<T>(gp, to_work<T>(a.backup.f[0][gi]), to_work<T>(a.backup.f[1][gi]),
                                   to_work<T>(a.backup.f[2][gi]), to_work<T>(a.backup.f[3][gi]),
                                   to_work<T>(a.backup.f[4][gi]));
            }
            const int o = in.pt.o;
            TS::put1f(sm, 0, o, ss.U);
            TS::put1f(sm, 1, o, ss.V);
            TS::put1f(sm, 2, o, ss.W);
            TS::put1f(sm, 3, o, ss.Tt);
            put2(sm, 4, o, s.ru, s.ru * ss.U + ss.p);
            put2(sm, 5, o, s.rv * ss.U, s.rw * ss.U);
            TS::put1f(sm, 6, o, (s.re + ss.p) * ss.U);
        });
    __syncthreads();
    if constexpr (SEG == kSeq)
        run_seq_tasks(sm.buf, sm.stride, TS::mail(sm), kSeqN1X, L, a.lgL, N, a.seg, a.h1, a.h2, 0, threadIdx.x);
    else if constexpr (SEG > 0)
        run_seg_x<SEG, FULL>(sm, P, L, N, a.seg, a.g1, a.g2, threadIdx.x, blockDim.x);
    else
        run_sweep_solves<2, PC>(sm, sizeof(T) == 4 ? kTasksX2 : kTasksX, 7, L, t.nlines, a.d1, a.d2, threadIdx.x,
                                blockDim.x, XDUM);
    __syncthreads();
    // phase C
    const T c43 = T(4.0 / 3.0), cpPr = (T)gp.cpPr, muref = (T)gp.mu_ref, slope = (T)0.76 * muref;
    struct InC { Pt pt; T v[4]; };
    batched<InC, sizeof(T) == 4 ? 4 : 2>(NL,
        [&](InC &in, int p) {
            in.pt = point<0, kXLineFirst>(t, p, L, P, a.lgL, a.divN, pad);
            const unsigned gi = in.pt.gi;
            in.v[0] = a.prim[0][gi]; in.v[1] = a.prim[1][gi]; in.v[2] = a.prim[2][gi]; in.v[3] = a.prim[4][gi];
        },
        [&](InC &in) {
            if (!in.pt.ok) return;
            const Pt &p = in.pt;
            const unsigned gi = p.gi;
            const Zn<T> zz = TS::z(a.d1, a.d2, p.n);
            const T U = in.v[0], V = in.v[1], W = in.v[2], Tt = in.v[3];
            T mu;
            if constexpr (kRecompute<T>) {
                mu = muref * visc_rpow(Tt) * Tt;
            } else {
                T rp;
                mu = muref * visc_powers(Tt, rp);
                a.mu[gi] = mu;
                a.amu[gi] = slope * rp;
            }
            T Ux, Uxx, Vx, Vxx, Wx, Wxx, Tx, Txx, cex, f1, f2, f3;
            TS::two(sm, 0, p, L, zz.z1, zz.z2, Ux, Uxx);
            TS::two(sm, 1, p, L, zz.z1, zz.z2, Vx, Vxx);
            TS::two(sm, 2, p, L, zz.z1, zz.z2, Wx, Wxx);
            TS::two(sm, 3, p, L, zz.z1, zz.z2, Tx, Txx);
            TS::two(sm, 4, p, L, zz.z1, zz.z1, cex, f1);
            TS::two(sm, 5, p, L, zz.z1, zz.z1, f2, f3);
            const T f4 = TS::one(sm, XF4, p, L, zz.z1);
            a.dx[0][gi] = Ux; a.dx[1][gi] = Vx; a.dx[2][gi] = Wx; a.dx[3][gi] = Tx;
            if (!PLAIN && a.tape[0]) {  // the tape's x entries (kIn* 0..16)
                T *const *g = a.tape;
                g[0][gi] = U; g[1][gi] = V; g[2][gi] = W; g[3][gi] = Tt;
                g[4][gi] = Ux; g[5][gi] = Vx; g[6][gi] = Wx; g[7][gi] = Tx;
                g[8][gi] = Uxx; g[9][gi] = Vxx; g[10][gi] = Wxx; g[11][gi] = Txx;
                g[12][gi] = cex; g[13][gi] = f1; g[14][gi] = f2; g[15][gi] = f3; g[16][gi] = f4;
            }
            a.R[0][gi] = -cex;
            // viscous terms of the momenta; their work is U, V, W times them
            const T v1 = mu * c43 * Uxx, v2 = mu * Vxx, v3 = mu * Wxx;
            a.R[1][gi] = v1 - f1;
            a.R[2][gi] = v2 - f2;
            a.R[3][gi] = v3 - f3;
            a.R[4][gi] = cpPr * mu * Txx + U * v1 + V * v2 + W * v3 - f4;
        });
}

// ---------------------------------------------------------------------
// sweep y
// ---------------------------------------------------------------------
enum { YU = 0, YU2, YV, YV2, YW, YW2, YT, YT2, YUX, YVX, YRV, YF1, YF2, YF3, YF4, YDUM, YNB2 };
constexpr int YNB = YDUM;
__constant__ Task kTasksY[8] = {{YU, YU, 0, YU, YU2, 1}, {YV, YV, 0, YV, YV2, 1}, {YW, YW, 0, YW, YW2, 1},
                                {YT, YT, 0, YT, YT2, 1}, {YUX, YUX, 0, YVX, YVX, 0},
                                {YRV, YRV, 0, YF1, YF1, 0}, {YF2, YF2, 0, YF3, YF3, 0},
                                {YF4, YF4, 0, YF4, YF4, 0}};
__constant__ Task kTasksY2[8] = {{YU, YU, 0, YU, YU2, 1}, {YV, YV, 0, YV, YV2, 1}, {YW, YW, 0, YW, YW2, 1},
                                 {YT, YT, 0, YT, YT2, 1}, {YUX, YUX, 0, YVX, YVX, 0},
                                 {YRV, YRV, 0, YF1, YF1, 0}, {YF2, YF2, 0, YF3, YF3, 0},
                                 {YF4, YF4, 0, YF4, YDUM, 0}};

// FP64: 3 blocks per SM (168 registers, no spills): 2.93 -> 2.67 ms per step at
// TGV 128^3, 37.5 -> 27.1 at HIT 256^3, the same bits
template <typename T, int PC, int SEG = 0, bool FULL = false, bool CL = false, bool WALL = false, int PLAIN = 0>
__global__ void __launch_bounds__(sweep_threads<T>(1), sizeof(T) == 4 ? kMinBlocksY : 3)
k_sweep_y(std::conditional_t<WALL, WallSweepArgs<T>, SweepArgs<T>> a) {
    using TS = TileOf<T, SEG>;
    constexpr bool SQ = SEG == kSeq;
    const int L = CL && !SQ ? kClLines : a.L, P = PC > 0 ? PC : a.P, lgL = CL && !SQ ? 5 : a.lgL;
    const int rank = CL ? (int)blockIdx.x % a.seg.C : 0;
    const Tile t = SQ ? make_seq_tile<1>(a.g, a.seg, L, rank)
                      : CL ? make_cluster_tile<1>(a.g, a.seg, rank) : make_tile<1>(a.g, L);
    const int N = t.N, NL = N * L, pad = FULL && !CL ? a.seg.pad : 0;
    const auto sm = TS::at(SQ ? kSeqN1Y : sizeof(T) == 4 ? YNB2 : YNB, L, P, SQ ? (a.seg.C > 1 ? a.seg.S : N) : CL ? 32 * a.seg.B : N, a.seg);
    struct InA { Pt pt; T v[11]; };
    batched<InA, sizeof(T) == 4 ? 4 : 2>(NL,
        [&](InA &in, int p) {
            in.pt = point<1>(t, p, L, P, lgL, a.divN, pad);
            const unsigned gi = in.pt.gi;
#pragma unroll
            for (int f = 0; f < 4; ++f) in.v[f] = a.qs[f + 1][gi];
#pragma unroll
            for (int f = 0; f < 5; ++f)
                if (f != 3 || !kRecompute<T>) in.v[4 + f] = a.prim[f][gi];
            in.v[9] = a.dx[0][gi];
            in.v[10] = a.dx[1][gi];
        },
        [&](InA &in) {
            if (!in.pt.ok) return;
            const int o = in.pt.o;
            const T ru = in.v[0], rv = in.v[1], rw = in.v[2], re = in.v[3];
            const T V = in.v[5];
            const T pp = kRecompute<T> ? pressure<T>(a.gas, ru, rv, rw, re, in.v[4], V, in.v[6]) : in.v[7];
            TS::put1f(sm, 0, o, in.v[4]);
            TS::put1f(sm, 1, o, V);
            TS::put1f(sm, 2, o, in.v[6]);
            TS::put1f(sm, 3, o, in.v[8]);
            put2(sm, 4, o, in.v[9], in.v[10]);
            put2(sm, 5, o, rv, ru * V);
            put2(sm, 6, o, rv * V + pp, rw * V);
            TS::put1f(sm, 7, o, (re + pp) * V);
        });
    if constexpr (CL) cluster_sync();
    else __syncthreads();
    if constexpr (SQ)
        run_seq_tasks(sm.buf, sm.stride, TS::mail(sm), kSeqN1Y, L, lgL, N, a.seg, a.h1, a.h2, rank, threadIdx.x);
    else if constexpr (WALL)
        run_cluster_tasks<FULL, 8, true, false, true>(sm.pair(0), sm.pstride / 2, cluster_mail(sm), a.seg, a.g1, a.g2,
                                                      rank, threadIdx.x, &a.w1, &a.w2);
    else if constexpr (CL)
        run_cluster_tasks<FULL, 8, true>(sm.pair(0), sm.pstride / 2, cluster_mail(sm), a.seg, a.g1, a.g2, rank,
                                         threadIdx.x);
    else if constexpr (SEG > 0)
        run_seg_tasks<SEG, FULL, 8, true>(sm, P, L, N, a.seg, a.g1, a.g2, threadIdx.x, blockDim.x);
    else
        run_sweep_solves<2, PC>(sm, sizeof(T) == 4 ? kTasksY2 : kTasksY, 8, L, t.nlines, a.d1, a.d2, threadIdx.x,
                                blockDim.x, YDUM);
    __syncthreads();
    const T c43 = T(4.0 / 3.0), c13 = T(1.0 / 3.0), cpPr = (T)a.gas.cpPr, muref = (T)a.gas.mu_ref;
    struct InC { Pt pt; T v[9]; };
    batched<InC, sizeof(T) == 4 ? kYConsumeBatch : 2>(NL,
        [&](InC &in, int p) {
            in.pt = point<1>(t, p, L, P, lgL, a.divN, pad);
            const unsigned gi = in.pt.gi;
            in.v[0] = a.prim[0][gi]; in.v[1] = a.prim[1][gi]; in.v[2] = a.prim[2][gi];
            in.v[3] = kRecompute<T> ? a.prim[4][gi] : a.mu[gi];
#pragma unroll
            for (int f = 0; f < 5; ++f) in.v[4 + f] = a.R[f][gi];
        },
        [&](InC &in) {
            if (!in.pt.ok) return;
            const Pt &p = in.pt;
            const unsigned gi = p.gi;
            const Zn<T> zz = TS::z(a.d1, a.d2, p.n);
            const T U = in.v[0], V = in.v[1], W = in.v[2];
            const T mu = kRecompute<T> ? muref * visc_rpow(in.v[3]) * in.v[3] : in.v[3];
            T Uy, Uyy, Vy, Vyy, Wy, Wyy, Ty, Tyy, Uxy, Vxy, cey, f1, f2, f3;
            TS::two(sm, 0, p, L, zz.z1, zz.z2, Uy, Uyy);
            TS::two(sm, 1, p, L, zz.z1, zz.z2, Vy, Vyy);
            TS::two(sm, 2, p, L, zz.z1, zz.z2, Wy, Wyy);
            TS::two(sm, 3, p, L, zz.z1, zz.z2, Ty, Tyy);
            TS::two(sm, 4, p, L, zz.z1, zz.z1, Uxy, Vxy);
            TS::two(sm, 5, p, L, zz.z1, zz.z1, cey, f1);
            TS::two(sm, 6, p, L, zz.z1, zz.z1, f2, f3);
            const T f4 = TS::one(sm, YF4, p, L, zz.z1);
            a.dy[0][gi] = Uy; a.dy[1][gi] = Vy; a.dy[2][gi] = Wy; a.dy[3][gi] = Ty;
            if (!PLAIN && a.tape[0]) {  // the tape's y entries (kIn* 17..31)
                T *const *g = a.tape;
                g[17][gi] = Uy; g[18][gi] = Vy; g[19][gi] = Wy; g[20][gi] = Ty;
                g[21][gi] = Uyy; g[22][gi] = Vyy; g[23][gi] = Wyy; g[24][gi] = Tyy;
                g[25][gi] = Uxy; g[26][gi] = Vxy; g[27][gi] = cey;
                g[28][gi] = f1; g[29][gi] = f2; g[30][gi] = f3; g[31][gi] = f4;
            }
            if constexpr (PLAIN != 0) {
                a.R[0][gi] = in.v[4] - cey;
            } else {
                int i, j, k;
                coords<1>(t, p.l, p.n, i, j, k);
                const int wd = a.wall_faces ? wall_dir(faces_of(a.g, i, j, k) & a.wall_faces) : -1;
                if (wd == 1) a.R[0][gi] = -cey;
                else if (wd < 0) a.R[0][gi] = in.v[4] - cey;
            }
            const T v1 = mu * (Uyy + c13 * Vxy), v2 = mu * (c43 * Vyy + c13 * Uxy), v3 = mu * Wyy;
            a.R[1][gi] = in.v[5] + (v1 - f1);
            a.R[2][gi] = in.v[6] + (v2 - f2);
            a.R[3][gi] = in.v[7] + (v3 - f3);
            a.R[4][gi] = in.v[8] + (cpPr * mu * Tyy + U * v1 + V * v2 + W * v3 - f4);
        });
}

// ---------------------------------------------------------------------
// sweep z + right-hand side + RK update
// ---------------------------------------------------------------------
enum { ZU = 0, ZU2, ZV, ZV2, ZW, ZW2, ZT, ZT2, ZS, ZWX, ZWY, ZRW, ZF1, ZF2, ZF3, ZF4, ZNB };
__constant__ Task kTasksZ[8] = {{ZU, ZU, 0, ZU, ZU2, 1}, {ZV, ZV, 0, ZV, ZV2, 1}, {ZW, ZW, 0, ZW, ZW2, 1},
                                {ZT, ZT, 0, ZT, ZT2, 1}, {ZS, ZS, 0, ZWX, ZWX, 0},
                                {ZWY, ZWY, 0, ZRW, ZRW, 0}, {ZF1, ZF1, 0, ZF2, ZF2, 0},
                                {ZF3, ZF3, 0, ZF4, ZF4, 0}};

// The z sweep's three phases as functions of (tile, shared-memory layout,
// thread range).
template <typename T, int PC, int SEG, bool FULL, bool CL, bool WALL, int PLAIN>
struct ZSweep {
    static constexpr bool SQ = SEG == kSeq;
    using TS = TileOf<T, SEG>;
    using SM = typename TS::SM;
    // A: stage the inputs of the 16 z-solves of tile t in sm
    static __device__ __forceinline__ void load(const SweepArgs<T> &a, const Tile &t, const SM &sm, int tid,
                                                int nthr) {
        const int L = CL && !SQ ? kClLines : a.L, P = PC > 0 ? PC : a.P, lgL = CL && !SQ ? 5 : a.lgL;
        const int NL = t.N * L, pad = FULL && !CL ? a.seg.pad : 0;
        struct InA { Pt pt; T v[13]; };
        batched<InA, sizeof(T) == 4 ? 4 : 2>(NL, tid, nthr,
            [&](InA &in, int p) {
                in.pt = point<2>(t, p, L, P, lgL, a.divN, pad);
                const unsigned gi = in.pt.gi;
#pragma unroll
                for (int f = 0; f < 4; ++f) in.v[f] = a.qs[f + 1][gi];
#pragma unroll
                for (int f = 0; f < 5; ++f)
                    if (f != 3 || !kRecompute<T>) in.v[4 + f] = a.prim[f][gi];
                in.v[9] = a.dx[0][gi];
                in.v[10] = a.dy[1][gi];
                in.v[11] = a.dx[2][gi];
                in.v[12] = a.dy[2][gi];
            },
            [&](InA &in) {
                if (!in.pt.ok) return;
                const int o = in.pt.o;
                const T ru = in.v[0], rv = in.v[1], rw = in.v[2], re = in.v[3];
                const T W = in.v[6];
                const T pp = kRecompute<T> ? pressure<T>(a.gas, ru, rv, rw, re, in.v[4], in.v[5], W) : in.v[7];
                TS::put1f(sm, 0, o, in.v[4]);
                TS::put1f(sm, 1, o, in.v[5]);
                TS::put1f(sm, 2, o, W);
                TS::put1f(sm, 3, o, in.v[8]);
                put2(sm, 4, o, in.v[9] + in.v[10], in.v[11]);
                put2(sm, 5, o, in.v[12], rw);
                put2(sm, 6, o, ru * W, rv * W);
                put2(sm, 7, o, rw * W + pp, (re + pp) * W);
            });
    }
    // B: the 16 solves (8 pairs) of every line of the tile
    static __device__ __forceinline__ void solve(const SweepArgs<T> &a, const Tile &t, const SM &sm, int tid,
                                                 int nthr, const WallOp *w1 = nullptr, const WallOp *w2 = nullptr) {
        const int rank = CL ? (int)blockIdx.x % a.seg.C : 0;
        if constexpr (SQ)
            run_seq_tasks(sm.buf, sm.stride, TS::mail(sm), kSeqN1Z, a.L, a.lgL, t.N, a.seg, a.h1, a.h2, rank, tid);
        else if constexpr (CL)
            run_cluster_tasks<FULL, 8, false, false, WALL>(sm.pair(0), sm.pstride / 2, cluster_mail(sm), a.seg, a.g1,
                                                           a.g2, rank, tid, w1, w2);
        else if constexpr (SEG > 0)
            run_seg_tasks<SEG, FULL, 8, false>(sm, PC > 0 ? PC : a.P, a.L, t.N, a.seg, a.g1, a.g2, tid, nthr);
        else
            run_sweep_solves<2, PC>(sm, kTasksZ, 8, a.L, t.nlines, a.d1, a.d2, tid, nthr, -1);
    }
    // C: right-hand side, dq and the RK update of every point of the tile
    static __device__ __forceinline__ void consume(const SweepArgs<T> &a, const Tile &t, const SM &sm, int tid,
                                                   int nthr) {
        const int L = CL && !SQ ? kClLines : a.L, P = PC > 0 ? PC : a.P, lgL = CL && !SQ ? 5 : a.lgL;
        const int NL = t.N * L, pad = FULL && !CL ? a.seg.pad : 0;
        const T c43 = T(4.0 / 3.0), c13 = T(1.0 / 3.0), c23 = T(2.0 / 3.0), cpPr = (T)a.gas.cpPr;
        const T muref = (T)a.gas.mu_ref;
        const double dt = *a.dt;
        const T dtw = (T)dt;
        const int st = a.rk_step;
        const bool tvd = PLAIN ? PLAIN == 2 : a.rk == 1;
        // which state arrays the update reads (uniform over the launch):
        //   qa = q1 (RK4 stage 1, all TVD-RK3 stages) or q2 (RK4 stages 2-4)
        //   qb = q1 for the FP64 RK4 qk update on stages 2-3, or the FP64 qk of
        //        TVD-RK3 stages 2-3
        //   mixed RK4: q2 accumulates every stage's increment in FP64; the next
        //   stage input qk = q1 + b dq exists only as an FP32 shadow, formed from
        //   q1's shadow (the stage input itself on stage 1)
        const bool use_q1a = tvd || st == 1;
        const bool need_qb = (!tvd && !a.mixed_rk4 && st > 1 && st < 4) || (tvd && st > 1);
        const bool need_q1s = a.mixed_rk4 && st > 1 && st < 4;
        const bool need_qs = a.mixed_rk4 && st == 1;
        // Right-hand side and update of a point in one pass: the FP64 additions
        // of the update (two an SM and clock) run under the other warps' FP32
        // work and loads.  As two passes over the tile, the update alone took 8.5 of a
        // block's 20 us at 128^3.
        struct InC {
            Pt pt;
            T v[18];
            double qa[5];
            double qb[5];  // FP64 state, or q1's FP32 shadow in the low word
        };
        batched<InC, 1>(NL, tid, nthr,
            [&](InC &in, int p) {
                in.pt = point<2>(t, p, L, P, lgL, a.divN, pad);
                const unsigned gi = in.pt.gi;
                in.v[0] = a.prim[0][gi]; in.v[1] = a.prim[1][gi]; in.v[2] = a.prim[2][gi];
                if constexpr (kRecompute<T>) {
                    in.v[3] = a.prim[4][gi];
                } else {
                    in.v[3] = a.mu[gi];
                    in.v[4] = a.amu[gi];
                }
#pragma unroll
                for (int f = 0; f < 4; ++f) { in.v[5 + f] = a.dx[f][gi]; in.v[9 + f] = a.dy[f][gi]; }
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    in.v[13 + f] = a.R[f][gi];
                    if constexpr (sizeof(T) == 4) {
                        in.qa[f] = use_q1a ? a.q1.f[f][gi] : a.q2.f[f][gi];
                        if (need_qs || need_q1s)
                            in.qb[f] = __hiloint2double(0, __float_as_int(need_qs ? a.qs[f][gi] : a.q1s[f][gi]));
                        else in.qb[f] = need_qb ? a.qk.f[f][gi] : 0.0;
                    } else {
                        in.qb[f] = need_qb ? (tvd ? a.qk.f[f][gi] : a.q1.f[f][gi]) : 0.0;
                        in.qa[f] = use_q1a ? a.q1.f[f][gi] : a.q2.f[f][gi];
                    }
                }
            },
            [&](InC &in) {
                if (!in.pt.ok) return;
                const Pt &p = in.pt;
                const unsigned gi = p.gi;
                const Zn<T> zz = TS::z(a.d1, a.d2, p.n);
                const T U = in.v[0], V = in.v[1], W = in.v[2];
                const T vz = kRecompute<T> ? muref * visc_rpow(in.v[3]) : T(0);
                const T mu = kRecompute<T> ? vz * in.v[3] : in.v[3], amu = kRecompute<T> ? (T)0.76 * vz : in.v[4];
                const T Ux = in.v[5], Vx = in.v[6], Wx = in.v[7], Tx = in.v[8];
                const T Uy = in.v[9], Vy = in.v[10], Wy = in.v[11], Ty = in.v[12];
                T Uz, Uzz, Vz, Vzz, Wz, Wzz, Tz, Tzz, S, Wxz, Wyz, cez, f1, f2, f3, f4;
                TS::two(sm, 0, p, L, zz.z1, zz.z2, Uz, Uzz);
                TS::two(sm, 1, p, L, zz.z1, zz.z2, Vz, Vzz);
                TS::two(sm, 2, p, L, zz.z1, zz.z2, Wz, Wzz);
                TS::two(sm, 3, p, L, zz.z1, zz.z2, Tz, Tzz);
                TS::two(sm, 4, p, L, zz.z1, zz.z1, S, Wxz);  // S = d/dz (Ux + Vy)
                TS::two(sm, 5, p, L, zz.z1, zz.z1, Wyz, cez);
                TS::two(sm, 6, p, L, zz.z1, zz.z1, f1, f2);
                TS::two(sm, 7, p, L, zz.z1, zz.z1, f3, f4);
                const T MuX = amu * Tx, MuY = amu * Ty, MuZ = amu * Tz;
                // shear rates, and the normal stresses 2 Ux - (2/3) div u
                const T s12 = Uy + Vx, s13 = Wx + Uz, s23 = Wy + Vz, dv = c23 * (Ux + Vy + Wz);
                const T g1 = T(2.0) * Ux - dv, g2 = T(2.0) * Vy - dv, g3 = T(2.0) * Wz - dv;
                // the viscous terms of the momenta: mu times second derivatives
                // and the viscosity gradient times the stresses; their work is
                // U, V, W times them, plus the dissipation
                const T w1 = mu * (Uzz + c13 * Wxz) + (MuX * g1 + MuY * s12 + MuZ * s13);
                const T w2 = mu * (Vzz + c13 * Wyz) + (MuY * g2 + MuX * s12 + MuZ * s23);
                const T w3 = mu * (c43 * Wzz + c13 * S) + (MuZ * g3 + MuX * s13 + MuY * s23);
                const T diss = Ux * g1 + Vy * g2 + Wz * g3 + (s12 * s12 + s13 * s13 + s23 * s23);
                T R[5];
                R[0] = in.v[13];
                R[1] = in.v[14] + (w1 - f1);
                R[2] = in.v[15] + (w2 - f2);
                R[3] = in.v[16] + (w3 - f3);
                R[4] = in.v[17] + (cpPr * (MuX * Tx + MuY * Ty + MuZ * Tz + mu * Tzz) +
                                   (U * w1 + V * w2 + W * w3 + mu * diss) - f4);
                // continuity and the post-step boundary fix-up (CSolver_AWS.cpp:1506-1679)
                bool zero_all = false, zero_mom = false;
                if constexpr (PLAIN) {
                    R[0] -= cez;
                } else {
                    int i, j, k;
                    coords<2>(t, p.l, p.n, i, j, k);
                    const int fc = faces_of(a.g, i, j, k);
                    const int wd = a.wall_faces ? wall_dir(fc & a.wall_faces) : -1;
                    if (wd == 2) R[0] = -cez;
                    else if (wd < 0) R[0] -= cez;
                    zero_all = (fc & a.sponge_kind_faces) != 0;
                    zero_mom = wd >= 0;
                }
                if (!PLAIN && a.diag[0]) {  // derivative fields of the last stage, for diagnostics
                    a.diag[0][gi] = Uz; a.diag[1][gi] = Vz; a.diag[2][gi] = Wz;
                }
                if (!PLAIN && a.tape[0]) {  // the tape's z entries (kIn* 32..47)
                    T *const *g = a.tape;
                    g[32][gi] = Uz; g[33][gi] = Vz; g[34][gi] = Wz; g[35][gi] = Tz;
                    g[36][gi] = Uzz; g[37][gi] = Vzz; g[38][gi] = Wzz; g[39][gi] = Tzz;
                    g[40][gi] = S; g[41][gi] = Wxz; g[42][gi] = Wyz; g[43][gi] = cez;
                    g[44][gi] = f1; g[45][gi] = f2; g[46][gi] = f3; g[47][gi] = f4;
                }
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    // plain form: dq = dt * RHS in FP64; mixed form: in FP32
                    T d = sizeof(T) == 8 ? (T)(dt * (double)R[f]) : dtw * R[f];
                    if (zero_all || (f > 0 && zero_mom)) d = T(0);
                    if (!PLAIN && a.dq_out[0]) a.dq_out[f][gi] = to_f64(d);
                    R[f] = d;
                }
                if (sizeof(T) == 8) {
                    // plain form: the reference's RK update in FP64
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        const double d = (double)R[f];
                        if (tvd) {  // TVD-RK3 (TVDRK3.hpp:38-96); qa = q1, qb = qk
                            if (st == 1) a.qk.f[f][gi] = in.qa[f] + d;
                            else if (st == 2) a.qk.f[f][gi] = 0.75 * in.qa[f] + 0.25 * in.qb[f] + 0.25 * d;
                            else a.q2.f[f][gi] = (1.0 / 3.0) * in.qa[f] + (2.0 / 3.0) * in.qb[f] + (2.0 / 3.0) * d;
                        } else {    // RK4 (RK4.hpp:35-118); qa = q1 (stage 1) or q2
                            const double ca = (st == 1 || st == 4) ? (1.0 / 6.0) : (1.0 / 3.0);
                            const double cb = (st == 3) ? 1.0 : 0.5;
                            a.q2.f[f][gi] = in.qa[f] + ca * d;
                            if (st == 1) a.qk.f[f][gi] = in.qa[f] + cb * d;
                            else if (st < 4) a.qk.f[f][gi] = in.qb[f] + cb * d;
                        }
                    }
                } else {
                    // mixed form: the FP32 increment accumulated into the FP64 state
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        const T d = R[f];
                        if (tvd) {
                            const double dd = to_f64(d);
                            double nv;
                            if (st == 1) { nv = in.qa[f] + dd; a.qk.f[f][gi] = nv; }
                            else if (st == 2) { nv = 0.75 * in.qa[f] + (0.25 * in.qb[f] + to_f64(T(0.25) * d)); a.qk.f[f][gi] = nv; }
                            else { nv = (1.0 / 3.0) * in.qa[f] + (2.0 / 3.0) * in.qb[f] + (2.0 / 3.0) * dd; a.q2.f[f][gi] = nv; }
                            if (a.shadow_target != SHADOW_NONE) a.shadow_out[f][gi] = narrow(nv);
                        } else {
                            // RK4: q2 += a_s dq in FP64 on every stage (RK4.hpp:35-118)
                            const T ca = (st == 1 || st == 4) ? T(1.0 / 6.0) : T(1.0 / 3.0);
                            const T cb = (st == 3) ? T(1.0) : T(0.5);
                            const double q2n = in.qa[f] + to_f64(ca * d);
                            a.q2.f[f][gi] = q2n;
                            if (st < 4) {
                                // the next stage input qk = q1 + cb*dq, kept as an FP32 shadow
                                a.shadow_out[f][gi] = fma(cb, d, (T)__int_as_float(__double2loint(in.qb[f])));
                            } else {
                                if (a.shadow_target == SHADOW_Q2) a.shadow_out[f][gi] = narrow(q2n);
                                // the filter's first pass input, q2 - fref in FP32
                                if (a.fluct_out) a.fluct[f][gi] = fluct_of(q2n, a.fref_hi[f], a.fref_lo[f]);
                            }
                        }
                    }
                }
            });
    }
};

// FP64: 3 blocks per SM (168 registers; 88 bytes of spill stores): 4.70 ->
// 4.52 ms per step at TGV 128^3, 52.5 -> 44.9 at HIT 256^3, the same bits
// PLAIN: as plain_kind below (x and y: 1 for either integrator)
template <typename T, int PC, int SEG = 0, bool FULL = false, bool CL = false, bool WALL = false, int PLAIN = 0>
__global__ void __launch_bounds__(sweep_threads<T>(2), sizeof(T) == 4 ? kMinBlocksZ : 3)
k_sweep_z(std::conditional_t<WALL, WallSweepArgs<T>, SweepArgs<T>> a) {
    using Z = ZSweep<T, PC, SEG, FULL, CL, WALL, PLAIN>;
    const int rank = CL ? (int)blockIdx.x % a.seg.C : 0;
    const Tile t = Z::SQ ? make_seq_tile<2>(a.g, a.seg, a.L, rank)
                         : CL ? make_cluster_tile<2>(a.g, a.seg, rank) : make_tile<2>(a.g, a.L);
    const auto sm = Z::TS::at(Z::SQ ? kSeqN1Z : ZNB, a.L, PC > 0 ? PC : a.P, Z::SQ ? (a.seg.C > 1 ? a.seg.S : t.N) : CL ? 32 * a.seg.B : t.N, a.seg);
    Z::load(a, t, sm, threadIdx.x, blockDim.x);
    if constexpr (CL) cluster_sync();
    else __syncthreads();
    if constexpr (WALL) Z::solve(a, t, sm, threadIdx.x, blockDim.x, &a.w1, &a.w2);
    else Z::solve(a, t, sm, threadIdx.x, blockDim.x);
    __syncthreads();
    Z::consume(a, t, sm, threadIdx.x, blockDim.x);
}

// ---------------------------------------------------------------------
// compact filter, one direction, five fields (Filter.cpp:98-171)
// ---------------------------------------------------------------------
// PC: the tile pitch as a compile-time constant (0: at run time); the mixed
// form's 128^3 pitches (x 9, y and z 8) are instantiated.
// Plain form: FP64 in, FP64 out, a.op = F.  Mixed form: a.op is the
// correction F - I, solved out of place (buffers 5..9), and the pass writes
// v + (F - I) v; the first pass reads FP64 q2 minus a per-field reference
// value (the field's initial mean, so the FP32 numbers are fluctuations), the
// middle pass works in FP32, and the last pass writes
// q1 = q2 + (filtered - unfiltered) in FP64 plus q1's FP32 shadow.
__constant__ Task kTasksF[3] = {{0, 0, 2, 1, 1, 2}, {2, 2, 2, 3, 3, 2}, {4, 4, 2, 4, 4, 2}};

// What a filter pass starts from: q2 itself (plain form), or its fluctuation.  One
// function for both kernels: the first and the last pass of a step may run different
// ones (a direction between walls), and q1 takes the difference of what they form.
template <typename T>
__device__ __forceinline__ T unfiltered(const FilterArgs<T> &a, int f, double q) {
    if constexpr (sizeof(T) == 8) return q;
    else return fluct_of(q, a.ref_hi[f], a.ref_lo[f]);
}

template <typename T, int DIR, int PC>
__global__ void __launch_bounds__(filter_threads<T>(), sizeof(T) == 4 ? kFilterMinBlocks : 4) k_filter(FilterArgs<T> a) {
    constexpr int B = sizeof(T) == 4 ? kFilterBatch : 2;
    constexpr bool kCorr = sizeof(T) == 4;
    const int L = a.L, P = PC > 0 ? PC : a.P;
    const Tile t = make_tile<DIR>(a.g, L);
    const int N = t.N, NL = N * L;
    Smem<T> sm = smem_layout<T>(kCorr ? 10 : 5, L, P, N);
    for (int p0 = threadIdx.x; p0 < NL; p0 += B * blockDim.x) {
        Pt pt[B];
        T v[B][5];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            pt[b] = point<DIR>(t, p0 + b * blockDim.x, L, P, a.lgL, a.divN);
            const unsigned gi = pt[b].gi;
#pragma unroll
            for (int f = 0; f < 5; ++f)
                v[b][f] = a.src64.f[f] ? unfiltered(a, f, a.src64.f[f][gi]) : a.src32[f][gi];
        }
#pragma unroll
        for (int b = 0; b < B; ++b) {
            if (!pt[b].ok) continue;
#pragma unroll
            for (int f = 0; f < 5; ++f) sm.b(f)[pt[b].o] = v[b][f];
        }
    }
    __syncthreads();
    if constexpr (kCorr) {
        // the five right-hand sides by the whole block, then one thread per
        // (field, line) for the recurrences alone
        rhs_pass<T, 4, 5>(sm, 0, 5, L, a.lgL, t.nlines, a.op);
        __syncthreads();
        for (int w = threadIdx.x; w < 5 * L; w += blockDim.x) {
            const int l = w & (L - 1), f = w >> a.lgL;
            if (l >= t.nlines) continue;
            thomas_inplace<T, PC>(sm.b(5 + f) + l, a.op, &sm.fact[(5 + f) * L + l], P);
        }
    } else {
        // plain form: one solve per thread, each field in place
        run_sweep_solves<4, 0>(sm, kTasksF, 3, L, t.nlines, a.op, a.op, (int)threadIdx.x, (int)blockDim.x);
    }
    __syncthreads();
    constexpr int BC = sizeof(T) == 4 ? kFilterConsumeBatch : 2;
    for (int p0 = threadIdx.x; p0 < NL; p0 += BC * blockDim.x) {
        Pt pt[BC];
        double q[BC][5];
        T u[BC][5];
#pragma unroll
        for (int b = 0; b < BC; ++b) {
            pt[b] = point<DIR>(t, p0 + b * blockDim.x, L, P, a.lgL, a.divN);
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                q[b][f] = a.delta_from.f[f] ? a.delta_from.f[f][pt[b].gi] : 0.0;
                u[b][f] = kCorr && a.unf[f] ? (T)a.unf[f][pt[b].gi] : T(0);
            }
        }
#pragma unroll
        for (int b = 0; b < BC; ++b) {
            if (!pt[b].ok) continue;
            const unsigned gi = pt[b].gi;
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                const T v = kCorr ? sm.b(f)[pt[b].o] + get(sm, 5 + f, pt[b], L, a.op) : get(sm, f, pt[b], L, a.op);
                if (a.dst64.f[f]) {
                    double nv;
                    if (a.delta_from.f[f]) {
                        // the unfiltered value: the first pass's FP32 input, or
                        // formed again from q2 (the same number either way)
                        const T v0 = kCorr && a.unf[f] ? u[b][f] : unfiltered(a, f, q[b][f]);
                        nv = q[b][f] + to_f64(v - v0);
                    } else {
                        nv = to_f64(v) + a.ref[f];
                    }
                    a.dst64.f[f][gi] = nv;
                    if (a.shadow_out[0]) a.shadow_out[f][gi] = narrow(nv);
                } else {
                    a.dst32[f][gi] = v;
                }
            }
        }
    }
}

// The mixed filter on periodic lines: the five fields' corrections by the
// segmented solves (cs3d_seg.cuh), added in place, so a tile is five buffers
// and the y and z tiles are 32 lines (128 bytes a row) wide.
// The plain form likewise, with F itself.
template <typename T, int DIR, int SEG, bool FULL>
__global__ void __launch_bounds__(sizeof(T) == 4 ? kFilterSegTpb : kFilterSegTpb64, sizeof(T) == 4 ? 2 : 3)
k_filter_seg(FilterArgs<T> a) {
    const int L = a.L, P = a.P;
    const Tile t = make_tile<DIR>(a.g, L);
    const int N = t.N, NL = N * L, pad = FULL ? a.seg.pad : 0;
    const int stride = seg_stride(N, P, a.seg.G, a.seg.pad);
    T *buf = reinterpret_cast<T *>(smem_raw);
    struct In { Pt pt; T v[5]; };
    batched<In, kFilterBatch>(NL,
        [&](In &in, int p) {
            in.pt = point<DIR>(t, p, L, P, a.lgL, a.divN, pad);
            const unsigned gi = in.pt.gi;
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                in.v[f] = a.src64.f[0] ? unfiltered(a, f, a.src64.f[f][gi]) : a.src32[f][gi];
            }
        },
        [&](In &in) {
            if (!in.pt.ok) return;
#pragma unroll
            for (int f = 0; f < 5; ++f) buf[f * stride + in.pt.o] = in.v[f];
        });
    __syncthreads();
    {
        const int lane0 = threadIdx.x & ((1 << a.seg.lgLW) - 1), seg = (threadIdx.x & 31) >> a.seg.lgLW;
        const int groups = max(1, L >> a.seg.lgLW);
        for (int u = threadIdx.x >> 5; u < 5 * groups; u += blockDim.x >> 5) {
            const int f = u / groups, l = ((u - f * groups) << a.seg.lgLW) + lane0;
            const bool active = l < L;
            seg_filter<SEG, FULL, sizeof(T) == 4>(seg_lane<SEG, FULL>(a.seg, buf + f * stride + (active ? l : 0), seg, N, P), P, a.sg,
                                  a.seg, lane0, active);
        }
    }
    __syncthreads();
    if constexpr (sizeof(T) == 8) {
        for (int p = threadIdx.x; p < NL; p += blockDim.x) {
            const Pt pt = point<DIR>(t, p, L, P, a.lgL, a.divN, pad);
            if (!pt.ok) continue;
#pragma unroll
            for (int f = 0; f < 5; ++f) (a.dst64.f[0] ? a.dst64.f[f] : a.dst32[f])[pt.gi] = buf[f * stride + pt.o];
        }
        return;
    } else {
    struct Out { Pt pt; double q[5]; float u[5]; };
    batched<Out, kFilterConsumeBatch>(NL,
        [&](Out &o, int p) {
            o.pt = point<DIR>(t, p, L, P, a.lgL, a.divN, pad);
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                o.q[f] = a.delta_from.f[0] ? a.delta_from.f[f][o.pt.gi] : 0.0;
                o.u[f] = a.unf[0] ? a.unf[f][o.pt.gi] : 0.f;
            }
        },
        [&](Out &o) {
            if (!o.pt.ok) return;
            const unsigned gi = o.pt.gi;
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                const float v = buf[f * stride + o.pt.o];
                if (a.dst64.f[0]) {
                    // q1 = q2 + (filtered - unfiltered); the unfiltered value is
                    // the first pass's FP32 input, or formed again from q2 (the
                    // same number either way)
                    const float v0 = a.unf[0] ? o.u[f] : unfiltered(a, f, o.q[f]);
                    const double nv = o.q[f] + widen(v - v0);
                    a.dst64.f[f][gi] = nv;
                    a.shadow_out[f][gi] = narrow(nv);
                } else {
                    a.dst32[f][gi] = v;
                }
            }
        });
    }
}

// ---------------------------------------------------------------------
// single operator on contiguous lines (Derivatives::calc1stDerivField etc.)
// ---------------------------------------------------------------------
__constant__ Task kTaskLone[1] = {{0, 0, 0, 0, 0, 0}};

template <int H>
__global__ void __launch_bounds__(128) k_line_op(LineOpArgs a) {
    const int L = a.L, N = a.op.N, P = a.P;
    const long long l0 = (long long)blockIdx.x * L;
    const int nl = (int)min((long long)L, a.nlines - l0);
    Smem<double> sm = smem_layout<double>(1, L, P, N);
    for (int p = threadIdx.x; p < N * L; p += blockDim.x) {
        const int l = p / N, n = p - l * N;
        if (l >= nl) continue;
        sm.b(0)[n * P + l] = a.in[(l0 + l) * N + n];
    }
    __syncthreads();
    // one solve per line (the task's duplicate second solve left out)
    run_sweep_solves<H, 0>(sm, kTaskLone, 1, L, nl, a.op, a.op, (int)threadIdx.x, (int)blockDim.x);
    __syncthreads();
    for (int p = threadIdx.x; p < N * L; p += blockDim.x) {
        Pt q;
        q.l = p / N;
        q.n = p - q.l * N;
        if (q.l >= nl) continue;
        q.o = q.n * P + q.l;
        a.out[(l0 + q.l) * N + q.n] = get(sm, 0, q, L, a.op);
    }
}

// ---------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------
template <typename T>
static size_t tile_smem(int nbuf, int L, int P, int N) {
    const int nf = (nbuf * L + 3) & ~3;
    return sizeof(T) * ((size_t)nf + (size_t)nbuf * buf_stride(N + kPad, P, L, (int)(sizeof(T) / 4)));
}

// The FP32-mixed sweeps' pair-interleaved tiles: the per-line factors, then
// (nbuf + 1) / 2 pair arrays of N rows each, then kPad rows of padding.  A
// solve's read-ahead past its line's end (up to kU + 1 rows, values never
// used) lands in the next pair array, or in the padding after the last one;
// no per-array padding, so that the mixed tiles fit the next-smaller shared
// memory carveout and leave L1 -- where the phases' global loads in flight
// are held -- more room (128^3: y and z 138.8 -> 133.4 kB a block, x
// 3 x 68.1 -> 3 x 65.8 kB).
static size_t pair_tile_smem(int nbuf, int L, int P, int N) {
    const int nf = (nbuf * L + 3) & ~3;
    return 4 * ((size_t)nf + (size_t)((nbuf + 1) / 2) * pair_stride(N, P) + (size_t)2 * kPad * P);
}

size_t planar_smem_bytes(int prec_bytes, int nbuf, int L, int P, int N) {
    return prec_bytes == 8 ? tile_smem<double>(nbuf, L, P, N) : tile_smem<float>(nbuf, L, P, N);
}
size_t sweep_smem_bytes(int prec_bytes, int nbuf, int L, int P, int N, const SegPlan *seg) {
    // the buffers and the mailboxes (a line's rows here: one block's, or all)
    if (prec_bytes == 8 && seg && seg->SEG)
        return 8 * (size_t)nbuf * (seq_stride(seg->C > 1 ? seg->S : N, L) + (seg->G == 1 ? 0 : 2 * (seg->C > 1 ? 1 : seg->G) * L));
    if (prec_bytes == 4 && seg && seg->C) return 8 * (8 * (size_t)(32 * seg->B) * kClLines + 16 * kClLines);
    if (prec_bytes == 4 && seg && seg->SEG && !seg->pair) return (size_t)XNB * 4 * seg_stride(N, P, seg->G, seg->pad);
    // segmented solves: the pair arrays alone (no line factors, no read-ahead)
    if (prec_bytes == 4 && seg && seg->SEG) return (size_t)((nbuf + 1) / 2) * 4 * seg_pair_stride(N, P, seg->G, seg->pad);
    return prec_bytes == 8 ? tile_smem<double>(nbuf, L, P, N) : pair_tile_smem(nbuf, L, P, N);
}
int sweep_nbuf(int dir, int prec_bytes) {
    if (prec_bytes == 4) return dir == 0 ? (int)XNB2 : dir == 1 ? (int)YNB2 : (int)ZNB;
    return dir == 0 ? (int)XNB : dir == 1 ? (int)YNB : (int)ZNB;
}
int sweep_ntask(int dir) { return dir == 0 ? 7 : 8; }
int filter_ntask() { return 3; }

template <typename K, typename A>
static cudaError_t launch_tile_kernel(K kernel, const A &a, dim3 grid, size_t sm, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    kernel<<<grid, a.threads, sm, s>>>(a);
    return cudaGetLastError();
}

static dim3 tile_grid(int dir, const Geom &g, int L) {
    if (dir == 0) return dim3((g.Ny + L - 1) / L, g.Nz);
    if (dir == 1) return dim3((g.Nx + L - 1) / L, g.Nz);
    return dim3((g.Nx + L - 1) / L, g.Ny);
}

// 1 (RK4) or 2 (TVD-RK3) where a launch has no walls, sponge faces, tape,
// diagnostics or increments to store, else 0.  An instance without their code
// has shorter load and update phases: 128^3 z 443 -> 425, y 238 -> 230, x 168 ->
// 164 us a step, 256^3 z 3.32 -> 3.20 ms, y 1.84 -> 1.78.  One instance per RK
// stage gave 454 and was dropped; between walls the same split gave nothing.
template <typename T>
static int plain_kind(const SweepArgs<T> &a) {
    if (a.wall_faces || a.sponge_kind_faces || a.diag[0] || a.tape[0] || a.dq_out[0]) return 0;
    return a.rk == 1 ? 2 : sizeof(T) == 8 || a.mixed_rk4 ? 1 : 0;
}

// the segmented instances: compile-time pitches for the full segments, the
// three segment lengths at run-time pitch for the others
static cudaError_t launch_seg_sweep(int dir, const SweepArgs<float> &a, dim3 grid, size_t sm, cudaStream_t s) {
    if (a.seg.C) {
        const bool f = a.seg.full;
        if (a.seg.wall) {
            WallSweepArgs<float> w;
            static_cast<SweepArgs<float> &>(w) = a;
            w.w1 = a.wall[0];
            w.w2 = a.wall[1];
            if (dir == 1) return launch_cluster(f ? k_sweep_y<float, 32, 32, true, true, true> : k_sweep_y<float, 32, 32, false, true, true>, w, grid, sm, s);
            return launch_cluster(f ? k_sweep_z<float, 32, 32, true, true, true> : k_sweep_z<float, 32, 32, false, true, true>, w, grid, sm, s);
        }
        const int plain = plain_kind(a);
#define CL_CASE(K, PL) return launch_cluster(f ? K<float, 32, 32, true, true, false, PL> : K<float, 32, 32, false, true, false, PL>, a, grid, sm, s)
        if (dir == 1) {
            if (plain) CL_CASE(k_sweep_y, 1);
            CL_CASE(k_sweep_y, 0);
        }
        if (plain == 1) CL_CASE(k_sweep_z, 1);
        if (plain == 2) CL_CASE(k_sweep_z, 2);
        CL_CASE(k_sweep_z, 0);
#undef CL_CASE
    }
#define SEG_CASE(K, PC, SEG, FULL) return launch_tile_kernel(K<float, PC, SEG, FULL>, a, grid, sm, s)
#define X_CASE(PC, SEG, FULL) \
    return plain_kind(a) ? launch_tile_kernel(k_sweep_x<float, PC, SEG, FULL, 1>, a, grid, sm, s) \
                         : launch_tile_kernel(k_sweep_x<float, PC, SEG, FULL>, a, grid, sm, s)
    if (a.seg.full) {
        if (dir == 0 && a.P == 17) X_CASE(17, 32, true);
        if (dir == 0 && a.P == 9) X_CASE(9, 32, true);
        if (dir == 0 && a.P == 5) X_CASE(5, 32, true);
        if (dir == 1 && a.P == 16) SEG_CASE(k_sweep_y, 16, 32, true);
        if (dir == 1 && a.P == 8) SEG_CASE(k_sweep_y, 8, 32, true);
        if (dir == 2 && a.P == 16) SEG_CASE(k_sweep_z, 16, 32, true);
        if (dir == 2 && a.P == 8) SEG_CASE(k_sweep_z, 8, 32, true);
        if (dir == 0) X_CASE(0, 32, true);
        if (dir == 1) SEG_CASE(k_sweep_y, 0, 32, true);
        SEG_CASE(k_sweep_z, 0, 32, true);
    }
    if (a.seg.SEG == 32) {
        if (dir == 0) X_CASE(0, 32, false);
        if (dir == 1) SEG_CASE(k_sweep_y, 0, 32, false);
        SEG_CASE(k_sweep_z, 0, 32, false);
    }
    if (a.seg.SEG == 24) {
        if (dir == 0) X_CASE(0, 24, false);
        if (dir == 1) SEG_CASE(k_sweep_y, 0, 24, false);
        SEG_CASE(k_sweep_z, 0, 24, false);
    }
    if (dir == 0) X_CASE(0, 16, false);
    if (dir == 1) SEG_CASE(k_sweep_y, 0, 16, false);
    SEG_CASE(k_sweep_z, 0, 16, false);
#undef SEG_CASE
#undef X_CASE
}

template <typename T>
cudaError_t launch_sweep(int dir, const SweepArgs<T> &a, cudaStream_t s) {
    const int N = dir == 0 ? a.g.Nx : dir == 1 ? a.g.Ny : a.g.Nz;
    const size_t sm = sweep_smem_bytes((int)sizeof(T), sweep_nbuf(dir, (int)sizeof(T)), a.L, a.P, N, &a.seg);
    const dim3 grid = tile_grid(dir, a.g, a.L);
    if constexpr (sizeof(T) == 4) {
        if (a.seg.SEG) return launch_seg_sweep(dir, a, grid, sm, s);
    } else if (a.seg.SEG == kSeq) {
        if (dir == 0) return launch_tile_kernel(k_sweep_x<T, 0, kSeq>, a, grid, sm, s);
        // the y sweep of this form gains nothing from it (2.31 against 2.32 ms)
        const int plain = plain_kind(a);
#define SEQ_CASE(K, PL) return launch_cluster(K<T, 0, kSeq, false, true, false, PL>, a, grid, sm, s)
        if (dir == 1) SEQ_CASE(k_sweep_y, 0);
        if (plain == 1) SEQ_CASE(k_sweep_z, 1);
        if (plain == 2) SEQ_CASE(k_sweep_z, 2);
        SEQ_CASE(k_sweep_z, 0);
#undef SEQ_CASE
    }
    if constexpr (sizeof(T) == 4) {
        if (dir == 0 && a.P == 9) return launch_tile_kernel(k_sweep_x<T, 9>, a, grid, sm, s);
        if (dir == 0 && a.P == 5) return launch_tile_kernel(k_sweep_x<T, 5>, a, grid, sm, s);
        if (dir == 1 && a.P == 16) return launch_tile_kernel(k_sweep_y<T, 16>, a, grid, sm, s);
        if (dir == 1 && a.P == 8) return launch_tile_kernel(k_sweep_y<T, 8>, a, grid, sm, s);
        if (dir == 2 && a.P == 16) return launch_tile_kernel(k_sweep_z<T, 16>, a, grid, sm, s);
        if (dir == 2 && a.P == 8) return launch_tile_kernel(k_sweep_z<T, 8>, a, grid, sm, s);
    }
    if (dir == 0) return launch_tile_kernel(k_sweep_x<T, 0>, a, grid, sm, s);
    if (dir == 1) return launch_tile_kernel(k_sweep_y<T, 0>, a, grid, sm, s);
    return launch_tile_kernel(k_sweep_z<T, 0>, a, grid, sm, s);
}

size_t filter_seg_smem(int prec_bytes, int L, int P, int N, const SegPlan &p) {
    return (size_t)5 * prec_bytes * seg_stride(N, P, p.G, p.pad);
}

template <int DIR, typename T>
static cudaError_t launch_filter_seg(const FilterArgs<T> &a, dim3 grid, size_t sm, cudaStream_t s) {
    if (a.seg.full) return launch_tile_kernel(k_filter_seg<T, DIR, 32, true>, a, grid, sm, s);
    if (a.seg.SEG == 32) return launch_tile_kernel(k_filter_seg<T, DIR, 32, false>, a, grid, sm, s);
    if (a.seg.SEG == 24) return launch_tile_kernel(k_filter_seg<T, DIR, 24, false>, a, grid, sm, s);
    return launch_tile_kernel(k_filter_seg<T, DIR, 16, false>, a, grid, sm, s);
}

template <typename T>
cudaError_t launch_filter(int dir, const FilterArgs<T> &a, cudaStream_t s) {
    const int N = dir == 0 ? a.g.Nx : dir == 1 ? a.g.Ny : a.g.Nz;
    if (a.seg.SEG) {
        const size_t fs = filter_seg_smem((int)sizeof(T), a.L, a.P, N, a.seg);
        const dim3 fg = tile_grid(dir, a.g, a.L);
        if (dir == 0) return launch_filter_seg<0>(a, fg, fs, s);
        if (dir == 1) return launch_filter_seg<1>(a, fg, fs, s);
        return launch_filter_seg<2>(a, fg, fs, s);
    }
    const size_t sm = tile_smem<T>(sizeof(T) == 4 ? 10 : 5, a.L, a.P, N);
    const dim3 grid = tile_grid(dir, a.g, a.L);
    if constexpr (sizeof(T) == 4) {
        if (dir == 0 && a.P == 9) return launch_tile_kernel(k_filter<T, 0, 9>, a, grid, sm, s);
        if (dir == 1 && a.P == 8) return launch_tile_kernel(k_filter<T, 1, 8>, a, grid, sm, s);
        if (dir == 2 && a.P == 8) return launch_tile_kernel(k_filter<T, 2, 8>, a, grid, sm, s);
    }
    if (dir == 0) return launch_tile_kernel(k_filter<T, 0, 0>, a, grid, sm, s);
    if (dir == 1) return launch_tile_kernel(k_filter<T, 1, 0>, a, grid, sm, s);
    return launch_tile_kernel(k_filter<T, 2, 0>, a, grid, sm, s);
}

cudaError_t launch_line_op(const LineOpArgs &a, cudaStream_t s) {
    const size_t sm = tile_smem<double>(1, a.L, a.P, a.op.N);
    const dim3 grid((unsigned)((a.nlines + a.L - 1) / a.L));
    if (a.op.H == 4) return launch_tile_kernel(k_line_op<4>, a, grid, sm, s);
    return launch_tile_kernel(k_line_op<2>, a, grid, sm, s);
}

template cudaError_t launch_sweep<double>(int, const SweepArgs<double> &, cudaStream_t);
template cudaError_t launch_sweep<float>(int, const SweepArgs<float> &, cudaStream_t);
template cudaError_t launch_filter<double>(int, const FilterArgs<double> &, cudaStream_t);
template cudaError_t launch_filter<float>(int, const FilterArgs<float> &, cudaStream_t);

}  // namespace cs3d
