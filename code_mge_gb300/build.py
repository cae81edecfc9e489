"""In-tree build of libmge_gpu.so for sm_103a (no CPU fallback exists).

The sources are compiled in parallel with nvcc and linked into
code_mge_gb300/_build/libmge_gpu.so.  The plain FP64 kernels are compiled
with --fmad=false so that no multiply-add is contracted: each expression
rounds exactly as the reference's Fortran evaluates it.
"""
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "_build")
LIB = os.path.join(OUT_DIR, "libmge_gpu.so")
ROOT = os.path.dirname(HERE)
# (source, object, its own flags); the kernels in three parts (MGE_PART), so
# that they compile side by side
SOURCES = [("mge_kernels.cu", "mge_kernels_f64.o", ["-DMGE_PART=0"]),
           ("mge_kernels.cu", "mge_kernels_f32.o", ["-DMGE_PART=1"]),
           ("mge_kernels.cu", "mge_kernels_group.o", ["-DMGE_PART=2"]),
           ("mge_runtime.cu", "mge_runtime.o", []),
           ("mge_noalloc.cu", "mge_noalloc.o", []),
           ("mge_restart.cpp", "mge_restart.o", [])]
HEADERS = ["mge_internal.h", "exact_ops.cuh", "fast_pow.cuh", "soft_fp64.cuh", "quick_quotient.h"]
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
NVCC_FLAGS = ["-std=c++17", "-O3", "--fmad=false", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-ffp-contract=off",
              "-I", os.path.join(ROOT, "include")]


def _nvcc():
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.isabs(c) and os.path.exists(c) or not os.path.isabs(c)):
            return c
    return "nvcc"


def _stale(out, deps):
    return not os.path.exists(out) or any(os.path.getmtime(out) < os.path.getmtime(d) for d in deps)


def build(force=False, verbose=False):
    os.makedirs(OUT_DIR, exist_ok=True)
    hdrs = [os.path.join(CSRC, h) for h in HEADERS] + [os.path.join(ROOT, "include", "mge_gpu.h")]
    objs, jobs = [], []
    for s, o, flags in SOURCES:
        src, obj = os.path.join(CSRC, s), os.path.join(OUT_DIR, o)
        objs.append(obj)
        if force or _stale(obj, [src] + hdrs):
            jobs.append([_nvcc()] + ARCH + NVCC_FLAGS + flags + ["-c", src, "-o", obj])

    def run(cmd):
        if verbose:
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + r.stdout + r.stderr)
        return r

    with ThreadPoolExecutor(max_workers=len(jobs) or 1) as ex:
        list(ex.map(run, jobs))
    if force or jobs or _stale(LIB, objs):
        run([_nvcc()] + ARCH + ["-shared", "-o", LIB + ".tmp"] + objs + ["-lcudart"])
        os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
