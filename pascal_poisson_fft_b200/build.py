"""Build recipe of libppf.so (sm_100a), in-tree next to this file.

Runs nvcc directly: one object per unit of UNITS, linked into a shared library
with a plain C ABI (include/ppf.h).  Usable without a GPU (cross-compiles).
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libppf.so")
CXX_OUT = os.path.join(HERE, "libppf_cxx.so")   # the C++ driver's solve calls on libppf
BUILD = os.path.join(HERE, "_build")
# (object, source, defines), the longest compilations first: the x and y
# transforms are split by element type and direction to build in parallel
UNITS = [("ppf_x_fwd32", "ppf_x.cu", ["-DPPF_REAL=float", "-DPPF_FWD=1"]),
         ("ppf_x_inv32", "ppf_x.cu", ["-DPPF_REAL=float", "-DPPF_FWD=0"]),
         ("ppf_batch", "ppf_batch.cu", []),
         ("ppf_x_fwd64", "ppf_x.cu", ["-DPPF_REAL=double", "-DPPF_FWD=1"]),
         ("ppf_x_inv64", "ppf_x.cu", ["-DPPF_REAL=double", "-DPPF_FWD=0"]),
         ("ppf_y_fwd32", "ppf_y.cu", ["-DPPF_REAL=float", "-DPPF_FWD=1"]),
         ("ppf_y_inv32", "ppf_y.cu", ["-DPPF_REAL=float", "-DPPF_FWD=0"]),
         ("ppf_y_fwd64", "ppf_y.cu", ["-DPPF_REAL=double", "-DPPF_FWD=1"]),
         ("ppf_y_inv64", "ppf_y.cu", ["-DPPF_REAL=double", "-DPPF_FWD=0"]),
         ("ppf_tdma", "ppf_tdma.cu", []), ("ppf_api", "ppf_api.cu", []), ("ppf_ghost", "ppf_ghost.cu", []),
         ("ppf_adjoint", "ppf_adjoint.cu", []), ("ppf_slab", "ppf_slab.cu", []), ("ppf_post", "ppf_post.cu", [])]
NVCC = os.environ.get("NVCC", "nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
         "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
         "-Xptxas", "-warn-spills"]


def _stale(obj: str, deps: list[str]) -> bool:
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    return any(os.path.getmtime(d) > t for d in deps)


def build(verbose: bool = False, jobs: int = min(8, os.cpu_count() or 4)) -> str:
    os.makedirs(BUILD, exist_ok=True)
    headers = [os.path.join(CSRC, h) for h in os.listdir(CSRC) if h.endswith((".cuh", ".h"))]
    headers.append(os.path.join(HERE, "..", "include", "ppf.h"))
    objs, todo = [], []
    for name, src, defs in UNITS:
        s = os.path.join(CSRC, src)
        o = os.path.join(BUILD, name + ".o")
        objs.append(o)
        if _stale(o, [s] + headers):
            todo.append((name, [NVCC, *FLAGS, *defs, "-c", s, "-o", o]))
    with ThreadPoolExecutor(max_workers=jobs) as pool:
        for _ in pool.map(lambda t: _compile(*t, verbose), todo):
            pass
    if _stale(OUT, objs):
        cmd = [NVCC, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", OUT, *objs, "-lcudart"]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.run(cmd, check=True)
    build_cxx_driver(verbose)
    return OUT


def build_cxx_driver(verbose: bool = False) -> str:
    """libppf_cxx.so: mpi_poisson::mpi_Poisson_FFT{1..5} of the C++ driver on
    libppf (g++; found next to libppf.so through its run path).  Its
    references to the driver's globals are resolved when the driver's
    program (or a test harness defining them) loads it."""
    src = os.path.join(CSRC, "ppf_cxx_driver.cpp")
    hdrs = [os.path.join(HERE, "..", "include", h) for h in ("ppf.h", "ppf_cxx_driver.h")]
    if _stale(CXX_OUT, [src, OUT] + hdrs):
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fopenmp",
               "-fvisibility=hidden", "-Wall", "-o", CXX_OUT, src, f"-L{HERE}", "-l:libppf.so",
               "-Wl,-rpath,$ORIGIN"]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.run(cmd, check=True)
    return CXX_OUT


def _compile(name: str, cmd: list[str], verbose: bool) -> None:
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
    text = r.stdout.decode(errors="replace")
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {name}:\n{text}")
    if text.strip():
        sys.stderr.write(text)


if __name__ == "__main__":
    print(build(verbose=True))
