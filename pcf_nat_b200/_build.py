"""Ahead-of-time build of the CUDA library for sm_100a (in-tree, plain nvcc, no torch headers).

Every .cu under csrc/ is compiled to an object of its own (in parallel, only when it or a header changed) and the
objects are linked into libna1d_b200.so next to this file. The autograd nodes (csrc/torch_nodes.cpp) are a Python extension of
their own, _na1d_torch.so, against the headers of the installed torch.
"""
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libna1d_b200.so")
NODES = os.path.join(PKG, "_na1d_torch.so")

NVCC_FLAGS = ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo"]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers():
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith((".cu", ".cpp"))] + [
        os.path.join(os.path.dirname(PKG), "include", "na1d_b200.h")]


def _deps():
    return sources() + _headers()


def is_stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(p) > t for p in _deps())


def build_library(force=False, verbose=False, extra_flags=()):
    """Compile every .cu under csrc/ and link libna1d_b200.so."""
    if not force and not is_stale():
        return LIB
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build libna1d_b200.so")
    os.makedirs(OBJ, exist_ok=True)
    newest_header = max(os.path.getmtime(p) for p in _headers())
    flags = NVCC_FLAGS + list(extra_flags)
    stamp = os.path.join(OBJ, "flags.txt")
    same_flags = os.path.exists(stamp) and open(stamp).read() == " ".join(flags)

    def compile_one(src):
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if (not force and same_flags and os.path.exists(obj) and
                os.path.getmtime(obj) >= max(os.path.getmtime(src), newest_header)):
            return obj
        cmd = [nvcc] + flags + ["-c", "-o", obj, src]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.check_call(cmd)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_one, sources()))
    open(stamp, "w").write(" ".join(flags))
    cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + objs
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.check_call(cmd)
    return LIB


def build_nodes(force=False, verbose=False):
    """Compile csrc/torch_nodes.cpp against the installed torch and link it to libna1d_b200.so (which has to exist)."""
    import torch
    root = os.path.dirname(os.path.abspath(torch.__file__))
    src = os.path.join(CSRC, "torch_nodes.cpp")
    stamp, version = os.path.join(OBJ, "torch.txt"), "%s %s" % (torch.__version__, sys.version)
    newest = max(os.path.getmtime(src), os.path.getmtime(os.path.join(os.path.dirname(PKG), "include", "na1d_b200.h")))
    if (not force and os.path.exists(NODES) and os.path.getmtime(NODES) >= newest and os.path.exists(stamp) and
            open(stamp).read() == version):
        return NODES
    cuda = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include"),
           sysconfig.get_path("include")]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI),
           "-DTORCH_EXTENSION_NAME=_na1d_torch", "-o", NODES, src] + [a for d in inc for a in ("-isystem", d)] + [
           "-L" + PKG, "-l:libna1d_b200.so", "-Wl,-rpath,$ORIGIN", "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cuda",
           "-ltorch_cpu", "-lc10_cuda", "-lc10", "-L" + os.path.join(cuda, "lib64"), "-lcublasLt"]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.check_call(cmd)
    open(stamp, "w").write(version)
    return NODES


if __name__ == "__main__":
    print(build_library(force=True, verbose=True))
    print(build_nodes(force=True, verbose=True))
