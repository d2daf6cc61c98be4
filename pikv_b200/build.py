"""Compile the CUDA sources under csrc/ into pikv_b200/libpikv_b200.so for sm_100a, and the native host module
csrc/host/host.cpp into pikv_b200/_host.so.

    python -m pikv_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU.  Objects go to csrc/build/, the shared
object next to this file, so it travels with the source tree.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(HERE, "libpikv_b200.so")
HOST = os.path.join(HERE, "_host.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

# no -use_fast_math: bit-exact codes need IEEE division and rint
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
    "-I", INCLUDE,
]


def nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the pikv_b200 CUDA library cannot be built")
    return exe


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _newest_header() -> float:
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return max(os.path.getmtime(h) for h in hs)


def _compile(src: str, force: bool, verbose: bool, ptxas_v: bool):
    obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
    if not force and os.path.exists(obj) and os.path.getmtime(obj) >= max(os.path.getmtime(src), _newest_header()):
        return obj, ""
    cmd = [nvcc(), *NVCC_FLAGS, "-c", src, "-o", obj]
    if ptxas_v:
        cmd[1:1] = ["-Xptxas", "-v"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{res.stdout}\n{res.stderr}")
    if verbose:
        print(" ".join(cmd))
    return obj, res.stderr


def build(force: bool = False, verbose: bool = False, ptxas_v: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    srcs = sources()
    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        results = list(ex.map(lambda s: _compile(s, force, verbose, ptxas_v), srcs))
    objs = [o for o, _ in results]
    if ptxas_v:
        for (_, log), s in zip(results, srcs):
            if log:
                print(f"==== {os.path.basename(s)}\n{log}")
    if force or not os.path.exists(LIB) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        cmd = [nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "--shared", "-o", LIB, *objs]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    _build_host(force)
    return LIB


def _build_host(force: bool) -> str:
    """The Python extension that marshals tensors for the library (needs torch's and Python's headers, no GPU)."""
    src = os.path.join(CSRC, "host", "host.cpp")
    newest = max(os.path.getmtime(f) for f in (src, os.path.join(INCLUDE, "pikv_b200.h")))
    if not force and os.path.exists(HOST) and os.path.getmtime(HOST) >= newest:
        return HOST
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(nvcc()))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(cuda, "include"), INCLUDE]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-I{d}" for d in inc), src, "-o", HOST, "-L" + os.path.join(root, "lib"), "-ltorch", "-ltorch_cpu", "-lc10",
           "-lc10_cuda", "-ltorch_python", "-L" + HERE, "-l:libpikv_b200.so", "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {src}:\n{res.stdout}\n{res.stderr}")
    return HOST


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    ap.add_argument("--ptxas-v", action="store_true", help="print registers / spills / shared memory per kernel")
    a = ap.parse_args()
    print(build(a.force, a.verbose, a.ptxas_v))
    sys.exit(0)
