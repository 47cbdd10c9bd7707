"""Build liblbm_gb300.so in-tree for sm_103a.

Translation units compiled in parallel and linked with nvcc:
  csrc/lbm_kernels.cu   device kernels (nvcc, sm_103a), once per type pair
  csrc/lbm_kernels2d.cu device kernels of the 2-D D2Q9 form (nvcc, sm_103a)
  csrc/lbm_capi.cu      the C ABI of include/lbm_gb300.h (nvcc host code)
  csrc/lbm_geometry.cu  device geometry precompute of a handle (explicitly
                        rounded float operations; built without contraction)
  csrc/lbm_geometry.cpp host geometry precompute of lbm_geometry_host (g++,
                        -ffp-contract=off so the float sequences match numpy
                        bit for bit)
  csrc/lbm_io.cpp       host output (the ASCII VTK writer)
Output: lbm/_lib/liblbm_gb300.so next to this file.
"""
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(ROOT, "csrc")
INCLUDE = os.path.join(os.path.dirname(ROOT), "include")
OUT_DIR = os.path.join(PKG, "_lib")
LIB = os.path.join(OUT_DIR, "liblbm_gb300.so")
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
HOST_FLAGS = "-fPIC,-ffp-contract=off"


def _nvcc():
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else (shutil.which("nvcc") or "nvcc")


def _sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC)
                  if f.endswith((".cu", ".cpp", ".cuh", ".h")))


def _stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = _sources() + [os.path.join(INCLUDE, "lbm_gb300.h"), os.path.abspath(__file__)]
    return any(os.path.getmtime(p) > t for p in deps)


def build(force=False, verbose=False):
    """Compile the library if a source is newer than it; return its path."""
    if not force and not _stale():
        return LIB
    os.makedirs(OUT_DIR, exist_ok=True)
    obj_dir = os.path.join(OUT_DIR, "obj")
    os.makedirs(obj_dir, exist_ok=True)
    nvcc = _nvcc()
    common = ["-O3", "-std=c++17", "-I", INCLUDE, "-I", CSRC]
    jobs = []
    # lbm_kernels.cu is compiled once per compute / storage type pair, in parallel
    cuda = [("lbm_kernels.cu", part) for part in range(3)]
    cuda += [(src, 0) for src in ("lbm_kernels2d.cu", "lbm_geometry.cu", "lbm_capi.cu")]
    for src, part in cuda:
        obj = os.path.join(obj_dir, f"{src}.{part}.o")
        # the 2-D kernels keep the reference's separate multiplies and adds
        # (no contraction into FMAs): their grids are small, and float32
        # parity with the reference is closer without contraction; the
        # geometry tables must be bit-exact
        extra = ["-fmad=false"] if src in ("lbm_kernels2d.cu", "lbm_geometry.cu") else []
        jobs.append([nvcc, *common, *ARCH, "-lineinfo", f"-DLBM_PART={part}", *extra, "-Xcompiler", HOST_FLAGS, "-c",
                     os.path.join(CSRC, src), "-o", obj])
    for src in ("lbm_geometry.cpp", "lbm_io.cpp"):
        obj = os.path.join(obj_dir, src + ".o")
        jobs.append([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-ffp-contract=off",
                     "-I", INCLUDE, "-I", CSRC, "-c", os.path.join(CSRC, src), "-o", obj])

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode:
            raise RuntimeError("compile failed: " + " ".join(cmd[-3:]))

    with ThreadPoolExecutor(len(jobs)) as ex:
        list(ex.map(run, jobs))
    objs = [j[-1] for j in jobs]
    tmp = LIB + ".tmp"
    run([nvcc, *ARCH, "-shared", "-o", tmp, *objs, "-lcudart", "-lpthread"])
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
