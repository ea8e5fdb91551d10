"""In-tree build of the CUDA library libcs3d_gb300.so (sm_103a only).

    python 3dcompactsolver_gb300/build.py [--force]

Compiles the translation units under csrc/ in parallel with nvcc and links
them into a shared library next to this file.  Rebuilds only when a source
is newer than the library.
"""
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INC = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "libcs3d_gb300.so")
OBJDIR = os.path.join(HERE, "_build")
SOURCES = ["cs3d_sweeps.cu", "cs3d_point.cu", "cs3d_abi.cu", "cs3d_adjoint.cu", "cs3d_lineop.cu"]
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
# --no-compress: the line information of the unrolled solves makes the device code large, and
# unpacking it took 24 ms of a process's first mixed step and 20 ms of its first adjoint (3 and 5
# so; a library of 51 instead of 15 MB)
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "--no-compress", "-Xcompiler", "-fPIC", "-Xcompiler", "-Wno-enum-compare",
         f"-I{INC}"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def _deps():
    out = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]
    out.append(os.path.join(INC, "cs3d.h"))
    return out


def up_to_date():
    if not os.path.exists(LIB):
        return False
    t = os.path.getmtime(LIB)
    return all(os.path.getmtime(d) <= t for d in _deps())


def build(force=False, verbose=False):
    """Compile and link the library; returns its path."""
    if not force and up_to_date():
        return LIB
    os.makedirs(OBJDIR, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src):
        obj = os.path.join(OBJDIR, os.path.splitext(src)[0] + ".o")
        cmd = [nvcc] + ARCH + FLAGS + ["-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{' '.join(cmd)}\n{r.stdout}{r.stderr}")
        if verbose and (r.stdout or r.stderr):
            print(r.stdout + r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    tmp = LIB + ".tmp"
    cmd = [nvcc] + ARCH + ["-shared", "-o", tmp] + objs
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{' '.join(cmd)}\n{r.stdout}{r.stderr}")
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose=True)
    print(path)
