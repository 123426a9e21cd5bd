"""Build libommx_b200.so (nvcc, sm_100a) and the Python host module _host.so (g++) in-tree.

    python -m open_ommx_serve_b200.build          # rebuild what is older than its sources

The library is plain CUDA C++ behind a C ABI (include/ommx_b200.h); it links nothing from torch.  _host.so is the
Python entry points' native half: it reads torch tensors and calls that ABI.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

from ._lib import HOST_MARK, HOST_PATH, host_built_for, host_target

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libommx_b200.so")
SOURCES = ("ommx_stage1_h8.cu", "ommx_stage1_h4.cu", "ommx_stage1_h2.cu", "ommx_stage1_h1.cu", "ommx_decode.cu", "ommx_pack.cu",
           "ommx_capi.cu")
HEADERS = ("ommx_common.cuh", "ommx_stage1.cuh", "ommx_decode_tc.cuh", "ommx_tables.inc", os.path.join("..", "..", "include", "ommx_b200.h"))
OBJ = os.path.join(PKG, "build")
HOST_LIB = HOST_PATH
HOST_SOURCE = os.path.join(CSRC, "ommx_host.cpp")
NVCC_FLAGS = ("-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
              "--no-compress")               # a process's first decode call waits 7 ms longer for the kernels of a compressed file


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def _older(target: str, sources) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(f) > os.path.getmtime(target) for f in sources)


def needs_build() -> bool:
    return _older(LIB, [os.path.join(CSRC, f) for f in SOURCES + HEADERS])


def _run(cmd) -> str:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("the build failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    return res.stderr


def build_host(force: bool = False) -> str:
    """Compile ``_host.so`` against the torch that this interpreter imports, unless it is newer than its sources and was built
    for this torch and python; returns its path."""
    import torch
    target = host_target()
    if not force and not _older(HOST_LIB, (HOST_SOURCE, os.path.join(PKG, "..", "include", "ommx_b200.h"))) and host_built_for(HOST_LIB) == target:
        return HOST_LIB
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    _run([os.environ.get("CXX") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC",
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DOMMX_HOST_BUILT_FOR="{HOST_MARK.decode()}{target}"',
          f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{sysconfig.get_paths()['include']}",
          f"-I{cuda}/include", "-o", HOST_LIB, HOST_SOURCE, f"-L{PKG}", "-l:" + os.path.basename(LIB),
          f"-L{root}/lib", "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"])
    return HOST_LIB


def _compile(source: str, force: bool, verbose: bool):
    """Object file of one CUDA source, rebuilt when it or a header is newer."""
    src, obj = os.path.join(CSRC, source), os.path.join(OBJ, source + ".o")
    if force or _older(obj, [src] + [os.path.join(CSRC, f) for f in HEADERS]):
        log = _run([_nvcc(), *NVCC_FLAGS, *(("-Xptxas", "-v") if verbose else ()), "-c", "-o", obj, src])
        if verbose:
            sys.stderr.write(log)
    return obj


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the CUDA sources (side by side) into ``libommx_b200.so`` next to this file and ``_host.so`` beside it;
    returns the library's path."""
    if force or needs_build():
        os.makedirs(OBJ, exist_ok=True)
        with ThreadPoolExecutor(len(SOURCES)) as pool:
            objs = list(pool.map(lambda f: _compile(f, force, verbose), SOURCES))
        _run([_nvcc(), *NVCC_FLAGS, "-shared", "-o", LIB, *objs])
    build_host(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
