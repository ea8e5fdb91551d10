"""The plain form's sequential line solves (as tests/test_seq_tasks_cpu.py: one
thread of the host for each thread of the blocks) under the thread sanitizer:
between two barriers no thread, idle ones among them, touches what another
writes."""
import os
import subprocess

import pytest

from conftest import ROOT
from test_seq_tasks_cpu import CSRC, MAIN, SHIM, _between

# Each barrier is used once: through one used again, a late thread would also wait for
# what the others did before they reached it the next time.
ARRIVE = r"""
#include <map>
#include <memory>
#include <mutex>
static std::mutex lock;
static std::map<std::pair<int, int>, std::unique_ptr<pthread_barrier_t>> bars;
static thread_local int phase;
static void arrive(pthread_barrier_t *bar, int first) {
    const bool cluster = bar == &cluster_bar;
    pthread_barrier_t *b;
    {
        std::lock_guard<std::mutex> g(lock);
        auto &e = bars[{cluster ? -1 : t_block, phase++}];
        if (!e) {
            e.reset(new pthread_barrier_t);
            pthread_barrier_init(e.get(), nullptr, (unsigned)(cluster ? place.size() : place.size() / smem.size()));
        }
        b = e.get();
    }
    pthread_barrier_wait(b);
}
"""

RUN = r"""
#include <cstdlib>
int main(int, char **a) {
    const int N = atoi(a[1]), d = atoi(a[2]), L = atoi(a[3]), n1 = d == 0 ? 9 : d == 1 ? 11 : 12;
    std::vector<double> f((size_t)n1 * L * N, 1.5), out((size_t)(n1 + 4) * L * N);
    return solve(N, d, L, n1, d == 0 ? 256 : 128, 0.1, f.data(), out.data());
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("race")
    abi = open(os.path.join(CSRC, "cs3d_abi.cu")).read()
    host = (_between(abi, "struct HostOp {", "// The filter's correction operator")
            + _between(abi, "// How a periodic line of N points is cut", "// The walls' rows of such a line"))
    seg = open(os.path.join(CSRC, "cs3d_seg.cuh")).read()
    for f in ("void cluster_sync(", "E *cluster_map("):
        seg = seg.replace(" " + f, " " + f[:-1] + "_ptx(")
    a, b = MAIN.index("static void arrive("), MAIN.index("void __syncwarp()")
    main = (MAIN[:a] + ARRIVE + MAIN[b:]).replace("@HOST@", host)
    (d / "cuda_runtime.h").write_text(SHIM)
    (d / "cs3d_seg.cuh").write_text(seg)
    (d / "main.cpp").write_text(main + RUN)
    exe = d / "race"
    r = subprocess.run(["g++", "-O0", "-g", "-std=c++17", "-w", "-pthread", "-fsanitize=thread", "-I", str(d), "-I", CSRC,
                        "-I", os.path.join(ROOT, "include"), str(d / "main.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    if r.returncode and "tsan" in r.stderr:
        pytest.skip("no thread sanitizer")
    assert r.returncode == 0, r.stderr
    return str(exe)


# one block in one, two and four segments, clusters of two and three; all have idle lanes
@pytest.mark.parametrize("d,N,L", [(0, 16, 8), (0, 81, 8), (0, 163, 4), (1, 64, 8), (1, 83, 8), (2, 161, 2)])
def test_no_access_races(program, d, N, L):
    r = subprocess.run([program, str(N), str(d), str(L)], capture_output=True, text=True, timeout=120)
    if "unexpected memory mapping" in r.stderr:
        pytest.skip("the thread sanitizer does not run here")
    assert "data race" not in r.stderr, r.stderr[:2000]
    assert r.returncode == 0, r.stderr[:2000]
