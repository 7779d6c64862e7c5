"""Builds libagd_b200.so (the CUDA kernels and the C ABI of include/agd_b200.h)
in-tree for sm_100a with nvcc."""
import os
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libagd_b200.so")
SOURCES = ["capi.cu", "eikonal.cu", "geodesic.cu", "adjoint.cu", "unet.cu",
           # the eikonal solve's kernels, by family (families.cuh)
           "solve_factor.cu", "solve_order2.cu", "solve_base.cu", "solve_rander.cu", "solve_order2f.cu",
           "solve_diagonal.cu", "solve_mpmix.cu", "solve_mp.cu", "solve_riemann2.cu", "solve_riemann3.cu",
           "solve_iso.cu"]
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ARCH_FLAGS + ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler",
                           "-fvisibility=hidden", "-I" + os.path.join(REPO, "include")]


def nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def build(verbose=False, extra=()):
    """Compiles every source to an object, several at a time, and links them."""
    srcs = [os.path.join(CSRC, s) for s in SOURCES]
    newest = max(os.path.getmtime(p) for p in srcs + [os.path.join(REPO, "include", f) for f in
                                                      ("agd_b200.h", "agd_warmstart.h")] +
                 [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))])
    if os.path.exists(LIB) and os.path.getmtime(LIB) >= newest and not extra:
        return LIB

    def run(cmd):
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.check_call(cmd)

    with tempfile.TemporaryDirectory() as tmp:
        objs = [os.path.join(tmp, os.path.basename(s) + ".o") for s in srcs]
        with ThreadPoolExecutor(max_workers=min(len(srcs), os.cpu_count() or 1)) as pool:
            list(pool.map(lambda so: run([nvcc()] + NVCC_FLAGS + list(extra) + ["-c", so[0], "-o", so[1]]),
                          zip(srcs, objs)))
        run([nvcc()] + ARCH_FLAGS + ["-shared"] + objs + ["-o", LIB + ".tmp"])
    os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    build(verbose=True, extra=tuple(sys.argv[1:]))
