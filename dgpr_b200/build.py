"""Builds the in-tree native library dgpr_b200/_lib/libdgb200.so (and the
dgb command-line driver) with nvcc for sm_100a.  No JIT, no torch extension:
the shared object sits in the source tree so it travels with the repository."""
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "_lib")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-O3",
         "--expt-relaxed-constexpr"]
# compiled once for the dispatch and once for the kernels of each order P = p + 1 (csrc/orders.hpp)
BY_ORDER = ["kernels_fp64.cu", "kernels_fp32.cu", "kernels_heat_fp64.cu", "kernels_heat_fp32.cu", "vspace_fp64.cu",
            "vspace_fp32.cu", "vspace_heat_fp64.cu", "vspace_heat_fp32.cu", "vspace_visc.cu", "adjoint.cu", "adjoint_heat.cu",
            "adjoint_gauss.cu", "adjoint_gauss_heat.cu", "residual_line.cu"]
SOURCES = ["host.cpp", "io.cpp", "checkpoint.cpp", "capi.cu", "vspace_tc.cu", "noalloc.cu", "check.cu", "adjoint_capi.cu",
           "geometry.cu"] + BY_ORDER


def _nvcc():
    for c in (os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc"), "nvcc"):
        if os.path.sep not in c or os.path.exists(c):
            return c
    return "nvcc"


def units():
    """(source, object, defines) of every translation unit, the longest first."""
    out = [(s, f"{s}.P{P}.o", [f"-DDGB_ORDER={P}"]) for P in range(7, 0, -1) for s in BY_ORDER]
    return out + [(s, s + ".o", []) for s in SOURCES]


def build(verbose=False, jobs=None):
    os.makedirs(LIB, exist_ok=True)
    headers = [os.path.join(CSRC, h) for h in os.listdir(CSRC) if h.endswith((".hpp", ".cuh"))]
    headers += [os.path.join(HERE, "..", "include", h) for h in ("dgb200.h", "dgb200_check.h")]
    newest = max(os.path.getmtime(h) for h in headers)

    def compile_unit(unit):
        src, obj, defines = unit
        src, obj = os.path.join(CSRC, src), os.path.join(LIB, obj)
        if os.path.exists(obj) and os.path.getmtime(obj) >= max(os.path.getmtime(src), newest):
            return obj
        cmd = [_nvcc()] + ARCH + FLAGS + defines + (["-x", "cu"] if src.endswith(".cpp") else []) + ["-c", src, "-o", obj]
        if verbose:
            print(" ".join(cmd), flush=True)
        p = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
        if p.returncode != 0:
            sys.stderr.write(p.stdout.decode())
            raise RuntimeError(f"nvcc failed on {os.path.basename(obj)}")
        if verbose and p.stdout:
            sys.stdout.write(p.stdout.decode())
        return obj

    with ThreadPoolExecutor(jobs or os.cpu_count()) as pool:
        objs = list(pool.map(compile_unit, units()))
    so = os.path.join(LIB, "libdgb200.so")
    subprocess.check_call([_nvcc()] + ARCH + ["-shared", "-o", so] + objs + ["-lcudart"])
    main_src = os.path.join(CSRC, "dgb_main.cpp")
    if os.path.exists(main_src):
        exe = os.path.join(LIB, "dgb")
        subprocess.check_call([_nvcc()] + ARCH + FLAGS + ["-x", "cu", main_src, "-o", exe, "-L" + LIB,
                               "-ldgb200", "-Xlinker", "-rpath=$ORIGIN"])
    return so


if __name__ == "__main__":
    build(verbose="-v" in sys.argv)
