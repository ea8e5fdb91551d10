"""The plain form's sequential line solves (`run_seq_tasks`, csrc/cs3d_seg.cuh)
compiled for the host, one thread of the host for each thread of a block or of
a cluster's blocks, at the line lengths where their plan changes: the results
against the oracle, and every barrier reached by all threads through one place
of the program (CUDA defines a block's barrier in conditional code only where
the condition is the same for the whole block)."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, rel_err

CSRC = os.path.join(ROOT, "3dcompactsolver_gb300", "csrc")

SHIM = r"""
#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>
#define __device__
#define __host__
#define __forceinline__ inline
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct double2 { double x, y; };
using std::max;
using std::min;
inline float2 make_float2(float x, float y) { return {x, y}; }
template <typename T> T __ldg(const T *p) { return *p; }
template <typename T> T __shfl_sync(unsigned, T v, int) { return v; }
inline unsigned __float_as_uint(float f) { unsigned u; memcpy(&u, &f, 4); return u; }
inline float __uint_as_float(unsigned u) { float f; memcpy(&f, &u, 4); return f; }
inline int __double2hiint(double d) { long long u; memcpy(&u, &d, 8); return (int)(u >> 32); }
inline int __double2loint(double d) { long long u; memcpy(&u, &d, 8); return (int)u; }
inline double __hiloint2double(int h, int l) {
    const unsigned long long u = (unsigned long long)(unsigned)h << 32 | (unsigned)l;
    double d;
    memcpy(&d, &u, 8);
    return d;
}
inline float __frcp_rn(float x) { return 1.0f / x; }
inline float __frsqrt_rn(float x) { return (float)(1.0 / std::sqrt((double)x)); }
inline float __log2f(float x) { return std::log2(x); }
using std::exp2f; using std::log2f;
void __syncwarp();
void __syncthreads();
namespace cs3d {
void cluster_sync();
char *cluster_map_bytes(const void *p, int rank);
template <typename E> E *cluster_map(E *p, int rank) { return (E *)cluster_map_bytes(p, rank); }
}
"""

MAIN = r"""
#include <execinfo.h>
#include <pthread.h>
#include <thread>
#include <vector>
#include "cs3d.h"
#include "cs3d_seg.cuh"
using namespace cs3d;
namespace {
@HOST@
}
static thread_local int t_block, t_slot;
static std::vector<std::vector<double>> smem;
static std::vector<std::vector<void *>> place;  // where each thread called the barrier from
static std::vector<pthread_barrier_t> block_bar;
static pthread_barrier_t cluster_bar;
static int apart;
static void arrive(pthread_barrier_t *bar, int first) {
    void *fr[8] = {};
    backtrace(fr, 8);
    place[t_slot].assign(fr + 2, fr + 8);  // (from the barrier's caller on)
    pthread_barrier_wait(bar);
    if (place[t_slot] != place[first]) __sync_fetch_and_add(&apart, 1);
    pthread_barrier_wait(bar);
}
void __syncwarp() {}
void __syncthreads() { arrive(&block_bar[t_block], t_slot - t_slot % (int)(place.size() / smem.size())); }
namespace cs3d {
void cluster_sync() { arrive(&cluster_bar, 0); }
char *cluster_map_bytes(const void *p, int rank) {
    return (char *)smem[rank].data() + ((const char *)p - (const char *)smem[t_block].data());
}
}
// field[n1][L][N] -> out[n1 + 4][L][N]: n1 first derivatives, four second ones
extern "C" int solve(int N, int d, int L, int n1, int threads, double dh, const double *field, double *out) {
    const SegPlan p = seq_plan(N, d);
    const SeqOp o1 = seq_op(make_op(1, N, CS3D_PERIODIC_SOLVE, dh, 0.0), p);
    const SeqOp o2 = seq_op(make_op(2, N, CS3D_PERIODIC_SOLVE, dh, 0.0), p);
    const int C = p.C, B = C > 1 ? 1 : p.G, R = C > 1 ? p.S : N, stride = R * L + 1;
    if (seq_slots(n1, B, L) * L > threads) return -1;
    int lgL = 0;
    while ((1 << lgL) < L) lgL++;
    smem.assign(C, std::vector<double>((n1 + 4) * (size_t)(stride + 2 * B * L)));
    place.assign((size_t)C * threads, {});
    apart = 0;
    for (int r = 0; r < C; r++)
        for (int k = 0; k < n1 + 4; k++)
            for (int l = 0; l < L; l++)
                for (int n = C > 1 ? seg_row0(p, r) : 0, m = 0; m < (C > 1 ? seg_rows(p, r) : N); n++, m++)
                    smem[r][k * stride + m * L + l] = field[((k < n1 ? k : k - n1) * L + l) * N + n];
    block_bar.resize(C);
    for (auto &b : block_bar) pthread_barrier_init(&b, nullptr, threads);
    pthread_barrier_init(&cluster_bar, nullptr, C * threads);
    std::vector<std::thread> all;
    for (int s = 0; s < C * threads; s++)
        all.emplace_back([&, s] {
            t_slot = s;
            t_block = s / threads;
            double *tile = smem[t_block].data();
            run_seq_tasks(tile, stride, tile + (n1 + 4) * stride, n1, L, lgL, C > 1 ? seg_rows(p, t_block) : N, p, o1,
                          o2, t_block, s % threads);
        });
    for (auto &t : all) t.join();
    for (int r = 0; r < C; r++)
        for (int k = 0; k < n1 + 4; k++)
            for (int l = 0; l < L; l++)
                for (int n = C > 1 ? seg_row0(p, r) : 0, m = 0; m < (C > 1 ? seg_rows(p, r) : N); n++, m++)
                    out[(k * L + l) * N + n] = smem[r][k * stride + m * L + l];
    for (auto &b : block_bar) pthread_barrier_destroy(&b);
    pthread_barrier_destroy(&cluster_bar);
    return apart;
}
"""


def _between(text, first, last):
    a = text.index(first)
    return text[a:text.index(last, a)]


@pytest.fixture(scope="module")
def seq_lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("seq")
    abi = open(os.path.join(CSRC, "cs3d_abi.cu")).read()
    host = (_between(abi, "struct HostOp {", "// The filter's correction operator")
            + _between(abi, "// How a periodic line of N points is cut", "// The walls' rows of such a line"))
    seg = open(os.path.join(CSRC, "cs3d_seg.cuh")).read()
    for f in ("void cluster_sync(", "E *cluster_map("):  # (PTX: the host's stand in for them)
        assert seg.count(" " + f) == 1
        seg = seg.replace(" " + f, " " + f[:-1] + "_ptx(")
    (d / "cuda_runtime.h").write_text(SHIM)
    (d / "cs3d_seg.cuh").write_text(seg)
    (d / "main.cpp").write_text(MAIN.replace("@HOST@", host))
    so = d / "seq.so"
    subprocess.run(["g++", "-O0", "-g", "-std=c++17", "-shared", "-fPIC", "-w", "-pthread", "-I", str(d), "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), str(d / "main.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    dp = ctypes.POINTER(ctypes.c_double)
    lib.solve.argtypes = [ctypes.c_int] * 5 + [ctypes.c_double, dp, dp]
    return lib


# x: one, two and four segments in a block; y and z: one block, clusters of two
# to eight with equal and unequal rows
@pytest.mark.parametrize("d,N", [(0, N) for N in (8, 9, 79, 80, 81, 121, 159, 160, 161, 163)]
                         + [(1, N) for N in (8, 64, 79, 80, 81, 129, 193)] + [(2, N) for N in (8, 65, 83, 161, 257, 513)])
def test_seq_tasks(seq_lib, oracle, d, N):
    n1 = (9, 11, 12)[d]
    L = 2 if d and N > 200 else 8 if N < 160 or d else 4
    rng = np.random.default_rng(N + d)
    f = np.ascontiguousarray(rng.standard_normal((n1, L, N)) + 3.0)
    out = np.empty((n1 + 4, L, N))
    dh = 2.0 * math.pi / N
    dp = ctypes.POINTER(ctypes.c_double)
    apart = seq_lib.solve(N, d, L, n1, 256 if d == 0 else 128, dh, f.ctypes.data_as(dp), out.ctypes.data_as(dp))
    ref1 = oracle.line_op_port(1, 0, N, dh, 0.49, f.reshape(-1, N)).reshape(n1, L, N)
    ref2 = oracle.line_op_port(2, 0, N, dh, 0.49, f[:4].reshape(-1, N)).reshape(4, L, N)
    # FP64, as the operators' other comparisons with the oracle
    assert rel_err(out[:n1], ref1) <= 1e-13
    assert rel_err(out[n1:], ref2) <= 1e-13
    assert apart == 0
