"""Builds wuda_b200/libwuda_b200.so from csrc/*.cu with nvcc for sm_100a.

nvcc cross-compiles without a GPU, so this runs anywhere the CUDA toolkit is present.
The library links the static CUDA runtime and resolves the one driver function it needs
(cuTensorMapEncodeTiled) at run time, so it also loads where no driver is installed.

wuda_b200/_fast.<interpreter>-<torch>.so (csrc/fast_ops.cpp, g++) is the operators' native call path from Python; it is built against
the installed torch, which its name says, and loads the library's entry points by name.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libwuda_b200.so")
OBJ_DIR = os.path.join(HERE, "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr", "--extended-lambda",
]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(HERE, "..", "include", "wuda_b200.h"))
    return hs


def build_fast(force=False):
    import runpy
    import sysconfig
    import torch
    fast = os.path.join(HERE, runpy.run_path(os.path.join(HERE, "native_calls.py"))["file_name"]())   # (the package may not import yet)
    src = os.path.join(CSRC, "fast_ops.cpp")
    newest = max(os.path.getmtime(p) for p in (src, os.path.join(HERE, "..", "include", "wuda_b200.h")))
    if not force and os.path.exists(fast) and os.path.getmtime(fast) >= newest:
        return fast
    root = os.path.dirname(os.path.abspath(torch.__file__))
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cmd = ([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
            "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI] +
           ["-I" + p for p in (root + "/include", root + "/include/torch/csrc/api/include", cuda + "/include",
                               sysconfig.get_paths()["include"])] +
           [src, "-o", fast, "-L" + root + "/lib", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"])
    subprocess.check_call(cmd)
    return fast


def build(force=False, verbose=False):
    nvcc = os.environ.get("NVCC", "nvcc")
    os.makedirs(OBJ_DIR, exist_ok=True)
    hdr_mtime = max(os.path.getmtime(h) for h in headers())
    objs = []
    procs = []
    for src in sources():
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if (not force and os.path.exists(obj)
                and os.path.getmtime(obj) >= max(os.path.getmtime(src), hdr_mtime)):
            continue
        cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        procs.append((cmd, subprocess.Popen(cmd)))
    for cmd, p in procs:
        if p.wait() != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd))
    if procs or not os.path.exists(LIB):
        cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a"]
        subprocess.check_call(cmd)
    build_fast(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
