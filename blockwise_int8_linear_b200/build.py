"""Builds libbi8.so (the CUDA kernels and their C ABI) with nvcc for sm_100a, and _native.so (the host path between Python and
libbi8.so) with g++ against the installed torch's headers, both in-tree.

    python -m blockwise_int8_linear_b200.build [--force] [--verbose]

The libraries are placed next to this file so that they travel with the source tree; nothing is
installed into site-packages and no JIT cache is used.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libbi8.so")
NATIVE = os.path.join(HERE, "_native.so")
NATIVE_SOURCE = "torch_ops.cpp"
SOURCES = ["api.cu", "quantize.cu", "quantize_tile.cu", "gemm_generic.cu", "gemm_tc.cu", "gemm_tc_skinny.cu", "gemm_smallm.cu", "no_alloc.cu", "peer_reduce.cu", "peer_reduce_large.cu", "quantize_pre.cu", "column_sum.cu", "rope_cache.cu", "copy_rows.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    # IEEE arithmetic is part of the contract (bit-exact quantization): no fast-math
    "--fmad=true", "-Xptxas", "-v",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the bi8 library cannot be built")
    return exe


def _deps_mtime() -> float:
    paths = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(HERE, "..", "include", "bi8.h"), __file__]
    return max(os.path.getmtime(p) for p in paths)


def _newer(path: str, mtime: float) -> bool:
    return os.path.exists(path) and os.path.getmtime(path) >= mtime


def _run(cmd, what: str) -> str:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{what}:\n" + r.stdout + r.stderr)
    return r.stdout + r.stderr


def _compile_native() -> str:
    """Object file of the extension: it needs torch's headers and none of libbi8's."""
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    obj = os.path.join(OBJ, NATIVE_SOURCE.replace(".cpp", ".o"))
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
          "-isystem", os.path.join(root, "include"), "-isystem", os.path.join(root, "include", "torch", "csrc", "api", "include"),
          "-isystem", os.path.join(cuda, "include"), "-isystem", sysconfig.get_paths()["include"],
          "-c", os.path.join(CSRC, NATIVE_SOURCE), "-o", obj], f"g++ failed for {NATIVE_SOURCE}")
    return obj


def _link_native(obj: str) -> None:
    import torch
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    # torch's libraries are in the process before this one is imported; libbi8.so lies beside it
    _run(["g++", "-shared", "-o", NATIVE, obj, "-L" + HERE, "-l:libbi8.so", "-Wl,-rpath,$ORIGIN", "-L" + libs, "-ltorch_python", "-ltorch",
          "-ltorch_cpu", "-lc10", "-lc10_cuda"], "link of _native.so failed")


def sources():
    return [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def build(force: bool = False, verbose: bool = False) -> str:
    deps = _deps_mtime()
    if not force and _newer(LIB, deps) and _newer(NATIVE, deps):
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: str) -> str:
        if src == NATIVE_SOURCE:
            return _compile_native()
        obj = os.path.join(OBJ, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        log = _run(cmd, f"nvcc failed for {src}")
        with open(obj + ".log", "w") as f:
            f.write(" ".join(cmd) + "\n" + log)
        if verbose:
            print(log)
        return obj

    with ThreadPoolExecutor(max_workers=6) as ex:
        objs = list(ex.map(compile_one, [NATIVE_SOURCE] + sources()))
    _run([nvcc, "-shared", "-o", LIB, *objs[1:], "-cudart", "static"], "link failed")
    _link_native(objs[0])
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
