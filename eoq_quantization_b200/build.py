"""Compile libeoq_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU), and `_native.so`, the torch-facing
front of it, with the host compiler."""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libeoq_b200.so")
NATIVE = os.path.join(HERE, "_native.so")
SOURCES = ["abi.cu", "kernels.cu", "qmm.cu", "wire_encode.cu", "rans_host.cpp", "wire_host.cpp"]
HEADERS = ["eoq_internal.h", os.path.join("..", "..", "include", "eoq_b200.h")]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _older(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.exists(d) and os.path.getmtime(d) > t for d in deps)


def stale() -> bool:
    return _older(LIB, [os.path.join(CSRC, s) for s in SOURCES + HEADERS]) or _older(NATIVE, [os.path.join(CSRC, "torch_native.cpp")])


def _run(cmd, verbose: bool) -> None:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError(os.path.basename(cmd[0]) + " failed:\n" + r.stdout + r.stderr)


def _build_native(verbose: bool) -> None:
    import torch
    from torch.utils.cpp_extension import include_paths
    tlib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.join(os.path.dirname(os.path.dirname(nvcc())), "include")
    _run([shutil.which("g++") or "c++", "-shared", "-O2", "-std=c++17", "-fPIC", "-Wall",
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-I" + sysconfig.get_paths()["include"], "-I" + cuda]
         + ["-I" + p for p in include_paths()]
         + [os.path.join(CSRC, "torch_native.cpp"), "-o", NATIVE, "-L" + HERE, "-l:libeoq_b200.so", "-L" + tlib,
            "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10", "-Wl,-rpath,$ORIGIN"], verbose)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not stale():
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    heads = [os.path.join(CSRC, h) for h in HEADERS]
    jobs, objects = [], []
    for s in SOURCES:
        src, obj = os.path.join(CSRC, s), os.path.join(OBJ, s + ".o")
        objects.append(obj)
        if force or _older(obj, [src] + heads):
            jobs.append([nvcc(), "-c", "-O3", "-std=c++17", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a",
                         "-Xcompiler", "-fPIC,-O3,-Wall", "-Xptxas", "-v" if verbose else "-O3", "-o", obj, src])
    with concurrent.futures.ThreadPoolExecutor(max(1, len(jobs))) as pool:
        list(pool.map(lambda c: _run(c, verbose), jobs))
    _run([nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + objects + ["-lpthread"], verbose)
    _build_native(verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--all" in sys.argv or "-v" in sys.argv, verbose="-v" in sys.argv))
