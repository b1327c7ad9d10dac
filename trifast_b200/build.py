"""Builds ``libtrifast_b200.so`` (the C-ABI library) in-tree with nvcc for sm_100a, and
``libtrifast_b200_torch.so`` (the PyTorch operators on top of it) with the C++ compiler.

    python -m trifast_b200.build [--force] [--verbose]

Every ``csrc/*.cu`` file is compiled to an object next to it (``csrc/_obj/``) and
linked into ``trifast_b200/libtrifast_b200.so``; ``csrc/torch_ops.cpp`` is compiled against
the installed PyTorch and linked to it.  Objects are rebuilt when a source or header is newer.  No GPU is needed to build.
"""

from __future__ import annotations

import argparse
import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(CSRC, "_obj")
LIB = os.path.join(PKG, "libtrifast_b200.so")
OPS_SRC = os.path.join(CSRC, "torch_ops.cpp")
OPS_LIB = os.path.join(PKG, "libtrifast_b200_torch.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--expt-relaxed-constexpr", "--extended-lambda",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def _newest(paths) -> float:
    return max(os.path.getmtime(p) for p in paths)


def _ops_commands(nvcc: str, obj: str):
    """Compile and link commands of the operator library.

    It links the shared C++ runtime by its file name: a compiler that has only the static one
    (``libstdc++.a``) would put a second copy into the process beside PyTorch's, and the two
    disagree about the facets of a locale: the first error message with a number in it crashes.
    """
    import torch
    from torch.utils.cpp_extension import include_paths
    root = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    inc = [f for p in include_paths() + [os.path.join(root, "include")] for f in ("-isystem", p)]
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    compile_cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-Wall",
                   f"-D_GLIBCXX_USE_CXX11_ABI={abi}", *inc, "-c", OPS_SRC, "-o", obj]
    link_cmd = [os.environ.get("CXX", "g++"), "-shared", "-o", OPS_LIB, obj, "-L", PKG,
                "-l:libtrifast_b200.so", "-l:libstdc++.so.6", "-L", libs, "-lc10", "-lc10_cuda",
                "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-Wl,-rpath,$ORIGIN", "-Wl,-rpath," + libs]
    return compile_cmd, link_cmd


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile and link the library; returns its path."""
    nvcc = _nvcc()
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(os.path.dirname(PKG), "include", "*.h"))
    dep_time = _newest(headers + [os.path.abspath(__file__)])
    jobs = []
    objs = []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), dep_time):
            cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    # the operators, compiled beside the kernels (their link waits for the library)
    ops_obj = os.path.join(OBJ, "torch_ops.o")
    ops_compile, ops_link = _ops_commands(nvcc, ops_obj)
    ops_stale = force or not os.path.exists(ops_obj) or \
        os.path.getmtime(ops_obj) < max(os.path.getmtime(OPS_SRC), dep_time)
    if ops_stale:
        jobs.append(ops_compile)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    if jobs:
        with cf.ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for cmd, r in ex.map(run, jobs):
                if verbose or r.returncode:
                    sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr + "\n")
                if r.returncode:
                    raise RuntimeError(f"compiling {cmd[-3]} failed")
    if jobs or force or not os.path.exists(LIB) or os.path.getmtime(LIB) < _newest(objs):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    if ops_stale or not os.path.exists(OPS_LIB) or \
            os.path.getmtime(OPS_LIB) < max(os.path.getmtime(ops_obj), os.path.getmtime(LIB)):
        _, r = run(ops_link)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("linking the operator library failed")
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
