"""Builds libportdnn_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU), and
the extension module behind api.py (api.front_path()), with the host compiler against torch's headers.

Each source is compiled to its own object (in parallel, only when it or a header changed) and
the objects are linked into the shared library.

Usage: python -m portdnn_b200.build [--force] [--verbose]
"""
import glob
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

from .api import front_path

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "_obj")
LIB = os.path.join(HERE, "libportdnn_b200.so")
FRONT_SOURCE = os.path.join(CSRC, "front.cpp")
SOURCES = ["c_api.cu", "hbm_kernels.cu", "direct_conv.cu", "tc_gemm.cu", "winograd.cu", "norm_kernels.cu",
           "layout_kernels.cu", "padded_conv.cu", "depthwise_tile.cu", "simt_gemm.cu", "collective.cu"]
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
         "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _headers():
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))] + \
        [os.path.join(HERE, "..", "include", "portdnn_b200.h")]


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def needs_build():
    return _stale(LIB, [os.path.join(CSRC, s) for s in SOURCES] + _headers()) or _stale(front_path(), _front_deps())


def _front_deps():
    return [FRONT_SOURCE, os.path.join(HERE, "..", "include", "portdnn_b200.h")]


def _front_command():
    """The extension finds libportdnn_b200.so beside itself and torch's libraries in the running process."""
    import torch
    from torch.utils import cpp_extension
    includes = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(os.path.dirname(_nvcc()), "..", "include")]
    libdir = os.path.join(os.path.dirname(torch.__file__), "lib")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall",
            "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)] + \
        [f for i in includes for f in ("-isystem", i)] + \
        [FRONT_SOURCE, "-o", front_path(), "-L" + HERE, "-lportdnn_b200", "-L" + libdir, "-lc10", "-lc10_cuda", "-ltorch_cpu",
         "-ltorch_python", "-Wl,-rpath,$ORIGIN"]


def _run(cmd, verbose):
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed: %s" % " ".join(cmd))


def build(force=False, verbose=False):
    if not force and not needs_build():
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    nvcc, headers = _nvcc(), _headers()
    jobs = []
    for src in SOURCES:
        path, obj = os.path.join(CSRC, src), os.path.join(OBJ, src[:-3] + ".o")
        if force or _stale(obj, [path] + headers):
            jobs.append([nvcc] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", path, "-o", obj])
    with ThreadPoolExecutor(max_workers=max(1, min(len(jobs), os.cpu_count() or 1))) as pool:
        list(pool.map(lambda c: _run(c, verbose), jobs))
    objs = [os.path.join(OBJ, s[:-3] + ".o") for s in SOURCES]
    if jobs or _stale(LIB, objs):
        _run([nvcc, "-shared", "-cudart", "shared", "-Xcompiler", "-fPIC"] + objs + ["-ldl", "-o", LIB], verbose)
    if force or _stale(front_path(), _front_deps()):
        _run(_front_command(), verbose)
        for other in glob.glob(os.path.join(HERE, "_front.*so")):  # of another Python or torch
            if other != front_path():
                os.remove(other)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(LIB)
