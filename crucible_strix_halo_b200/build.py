"""Builds libcrucible_attn.so (sm_100a) in-tree with nvcc, and _binding.so (the host path of layers.py) with g++.

    python -m crucible_strix_halo_b200.build [--force]
"""
import concurrent.futures
import glob
import os
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libcrucible_attn.so")
BINDING = os.path.join(PKG, "_binding.so")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xptxas", "-O3"]


def _newer(dst, srcs):
    if not os.path.exists(dst):
        return False
    m = os.path.getmtime(dst)
    return all(os.path.getmtime(s) <= m for s in srcs)


def _run(cmd):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("command failed: %s\n%s\n%s" % (" ".join(cmd), r.stdout, r.stderr))
    return r.stdout + r.stderr


def build_library(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(ROOT, "include", "*.h"))
    if not force and _newer(LIB, sources + headers):      # a shipped library that is newer than every source
        return LIB
    jobs = []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if force or not _newer(obj, [src] + headers):
            jobs.append(["nvcc", *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-c", src, "-o", obj])
    with concurrent.futures.ThreadPoolExecutor(max_workers=8) as ex:
        for out in ex.map(_run, jobs):
            if verbose:
                print(out)
    objs = [os.path.join(OBJ, os.path.basename(s)[:-3] + ".o") for s in sources]
    if force or jobs or not os.path.exists(LIB):
        _run(["nvcc", "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, *objs, "-lcudart"])
    return LIB


def build_binding(force=False):
    """Needs the library and torch's headers; links against both (the library is found beside the binding)."""
    src = os.path.join(PKG, "native", "binding.cpp")
    if not force and _newer(BINDING, [src, os.path.join(ROOT, "include", "crucible_attn.h")]):
        return BINDING
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    libs = cpp_extension.library_paths(device_type="cuda")
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
          *["-I" + d for d in cpp_extension.include_paths(device_type="cuda") + [sysconfig.get_paths()["include"]]], src, "-o", BINDING,
          "-L" + PKG, "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN", *["-L" + d for d in libs], "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"])
    return BINDING


def build_all(force=False, verbose=False):
    build_library(force, verbose)
    build_binding(force)
    return LIB


if __name__ == "__main__":
    force = "--force" in sys.argv
    print(build_all(force, verbose="-v" in sys.argv))
