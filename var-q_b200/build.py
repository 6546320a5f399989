"""Build libvarq_b200.so (nvcc, sm_100a) and the host extension _host.so (g++, CPython over ATen) in-tree.

    python var-q_b200/build.py [--force] [--verbose]

The library is compiled straight into ``var-q_b200/VAR_Q/`` next to the Python
wrapper so that a checkout carries its binary along; nothing is installed into
site-packages and no JIT cache is used.
"""
import argparse
import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB_PATH = os.path.join(HERE, "VAR_Q", "libvarq_b200.so")
HOST_SRC = os.path.join(HERE, "csrc_host", "varq_host.cpp")
HOST_PATH = os.path.join(HERE, "VAR_Q", "_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-cudart", "static", "--threads", "0",
]


def find_nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: set NVCC or put it on PATH")


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def is_stale():
    if not os.path.exists(LIB_PATH):
        return True
    built = os.path.getmtime(LIB_PATH)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(INCLUDE, "*.h"))
    return any(os.path.getmtime(p) > built for p in deps)


def build_host(force=False, verbose=False):
    """Compile the host extension against the installed torch; it links to libvarq_b200.so next to it."""
    header = os.path.join(INCLUDE, "varq_b200.h")
    if not force and os.path.exists(HOST_PATH) and os.path.getmtime(HOST_PATH) > max(os.path.getmtime(HOST_SRC), os.path.getmtime(header)):
        return HOST_PATH
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda_home = os.path.dirname(os.path.dirname(find_nvcc()))
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", INCLUDE, "-I", sysconfig.get_paths()["include"], "-I", os.path.join(cuda_home, "include")]
    for p in cpp_extension.include_paths():
        cmd += ["-isystem", p]
    cmd += [HOST_SRC, "-o", HOST_PATH, "-L", os.path.dirname(LIB_PATH), "-l:libvarq_b200.so", "-Wl,-rpath,$ORIGIN", "-L", torch_lib,
            "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError("g++ failed building _host.so")
    return HOST_PATH


def build_library(force=False, verbose=False):
    """Compile every .cu of csrc/ into one shared library, and the host extension; returns the library's path."""
    if not force and not is_stale():
        build_host()
        return LIB_PATH
    cmd = [find_nvcc()] + NVCC_FLAGS + ["-I", INCLUDE, "-I", CSRC]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += sources() + ["-o", LIB_PATH]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed building libvarq_b200.so")
    build_host(force=force, verbose=verbose)
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build_library(force=a.force, verbose=a.verbose))
