"""Builds the CUDA library (libqlka.so, next to this file) for sm_100a with nvcc, and the torch binding over it
(_qlka_torch.so) with g++.

    python quasi-linear-kernel-attention_b200/build.py [--force] [--verbose]

The library is plain nvcc, no torch headers: its ABI is the C header include/qlka.h. The binding is the only file that
sees torch.
"""

import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libqlka.so")
SOURCES = ["qlka_api.cu", "sort_rank.cu", "sort_rank_large.cu", "walk_laplace.cu", "walk_prefix.cu", "walk_events.cu", "dense_tiles.cu", "dense_gradient.cu", "encoder_linear.cu", "aux_kernels.cu"]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
         "-Xcompiler", "-fPIC", "--threads", "4"]


BINDING = os.path.join(HERE, "_qlka_torch.so")
BINDING_SOURCE = os.path.join(CSRC, "torch_binding.cpp")
HEADER = os.path.join(HERE, "..", "include", "qlka.h")


def _stale(target, deps):
    return not os.path.exists(target) or any(os.path.getmtime(d) > os.path.getmtime(target) for d in [*deps, HEADER, os.path.abspath(__file__)])


def build_binding(force=False, verbose=False):
    """Compile the torch binding; returns the path."""
    if not force and not _stale(BINDING, [BINDING_SOURCE]):
        return BINDING
    import torch
    from torch.utils import cpp_extension
    libs = [d for d in cpp_extension.library_paths() if os.path.isdir(d)]
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-DTORCH_EXTENSION_NAME=_qlka_torch", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{d}" for d in [*cpp_extension.include_paths(), "/usr/local/cuda/include", sysconfig.get_paths()["include"]]],
           BINDING_SOURCE, "-o", BINDING, *[f"-L{d}" for d in libs], "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", "-ldl"]
    if verbose:
        print(" ".join(cmd))
    subprocess.check_call(cmd)
    return BINDING


def build(force=False, verbose=False):
    """Compile every .cu of csrc/ into libqlka.so, and the torch binding; returns the library's path."""
    build_binding(force, verbose)
    if not force and not _stale(LIB, [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))]):
        return LIB
    objs = []
    procs = []
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    for src in SOURCES:
        obj = os.path.join(HERE, "build", src.replace(".cu", ".o"))
        cmd = [NVCC, *FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            print(f"--- {src}\n{out}")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    subprocess.check_call([NVCC, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
