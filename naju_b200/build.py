"""In-tree build of libnaju_b200.so (hand-written sm_100a CUDA behind a C ABI) and of _native.so, the
CPython extension that is its host path.

    python -m naju_b200.build [--force]

nvcc cross-compiles for sm_100a without a GPU.  Both libraries land next to this file so they
travel with the source tree; nothing is written outside the package.
"""
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libnaju_b200.so")
NATIVE = os.path.join(HERE, "_native.so")

SOURCES = ["api.cu", "fwd_simt.cu", "fwd_chan.cu", "fwd_tc2.cu", "fwd_tc3.cu", "bwd_simt.cu", "bwd_chan.cu", "bwd_tc.cu", "fwd_wide.cu", "bwd_wide.cu", "step.cu", "fwd_noalloc.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-I", INCLUDE, "-I", CSRC]


def _newest(src=None):
    """Time stamp of the newest source: the headers and `src`, or every CUDA source."""
    names = [f for f in os.listdir(CSRC) if f.endswith((".cuh", ".h")) or f == src or (src is None and f.endswith(".cu"))]
    deps = [os.path.join(CSRC, f) for f in names] + [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return max(os.path.getmtime(f) for f in deps)


def _run(cmd, what):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")


def _up_to_date(path, src=None):
    return os.path.exists(path) and os.path.getmtime(path) >= _newest(src)


def _build_native():
    """Host compiler only: libtorch headers, linked against libnaju_b200.so beside it."""
    import torch
    tdir = os.path.dirname(torch.__file__)
    inc = [os.path.join(tdir, "include"), os.path.join(tdir, "include", "torch", "csrc", "api", "include"),
           os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"), sysconfig.get_paths()["include"], INCLUDE]
    obj = os.path.join(OBJ, "torch_host.o")
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-DTORCH_EXTENSION_NAME=_native", "-DTORCH_API_INCLUDE_EXTENSION_H",
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] +
         [a for i in inc for a in ("-isystem", i)] + ["-c", os.path.join(CSRC, "torch_host.cpp"), "-o", obj], "g++ torch_host.cpp")
    _run(["g++", "-shared", "-o", NATIVE, obj, "-L" + HERE, "-l:libnaju_b200.so", "-Wl,-rpath,$ORIGIN",
          "-L" + os.path.join(tdir, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"],
         "link of _native.so")


def _compile(src):
    obj = os.path.join(OBJ, src.replace(".cu", ".o"))
    if _up_to_date(obj, src):
        return obj
    _run(["nvcc"] + NVCC_FLAGS + ["-c", os.path.join(CSRC, src), "-o", obj], f"nvcc {src}")
    return obj


def build(force=False, verbose=False):
    """Compiles every CUDA source for sm_100a, links libnaju_b200.so and builds _native.so on top of it.
    Returns the library's path."""
    os.makedirs(OBJ, exist_ok=True)
    if force:
        for f in os.listdir(OBJ):
            if f.endswith(".o"):
                os.remove(os.path.join(OBJ, f))
    if force or not _up_to_date(LIB):
        with ThreadPoolExecutor(max_workers=min(len(SOURCES), os.cpu_count() or 1)) as ex:
            objs = list(ex.map(_compile, SOURCES))
        _run(["nvcc", "-shared", "-o", LIB] + objs, "link of libnaju_b200.so")
    # (_native.so calls the C ABI of include/naju_b200.h, so the library's own sources do not concern it)
    if force or not _up_to_date(NATIVE, "torch_host.cpp"):
        _build_native()
    if verbose:
        print("built", LIB, NATIVE)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
