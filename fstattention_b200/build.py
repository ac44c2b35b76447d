"""Build libfstattn_b200.so (nvcc, sm_100a) and the Python host module on top of it, in-tree.

  python -m fstattention_b200.build [--force]

One object per .cu file, compiled in parallel, then linked into
``fstattention_b200/libfstattn_b200.so``; ``csrc/fst_host.cpp`` becomes ``_fst_host.so`` (a CPython
extension against torch's headers, linked to the library).  Nothing is rebuilt when the outputs
are newer than every source file.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")
LIB = os.path.join(PKG, "libfstattn_b200.so")
HOST = os.path.join(PKG, "_fst_host.so")
HOST_SRC = os.path.join(CSRC, "fst_host.cpp")
OBJ = os.path.join(PKG, "build")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps():
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hdrs += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return hdrs


def up_to_date() -> bool:
    if not (os.path.exists(LIB) and os.path.exists(HOST)):
        return False
    t = min(os.path.getmtime(LIB), os.path.getmtime(HOST))
    return all(os.path.getmtime(p) <= t for p in sources() + _deps() + [HOST_SRC, os.path.abspath(__file__)])


def _build_host() -> None:
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if not cxx:
        raise RuntimeError("g++ not found; set CXX or put it on PATH")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = cpp_extension.include_paths() + [os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", INCLUDE, "-I", CSRC, *(x for d in inc for x in ("-isystem", d)), HOST_SRC, "-o", HOST,
           LIB, "-Wl,-rpath,$ORIGIN", "-L", lib, "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10",
           "-lc10_cuda", "-L", os.path.join(cuda, "lib64"), "-lcudart"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {HOST_SRC}:\n{res.stdout}\n{res.stderr}")


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB
    nvcc = _nvcc()
    os.makedirs(OBJ, exist_ok=True)
    newest_hdr = max(os.path.getmtime(p) for p in _deps())

    def compile_one(src):
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if (not force and os.path.exists(obj)
                and os.path.getmtime(obj) >= max(os.path.getmtime(src), newest_hdr)):
            return obj
        cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{res.stdout}\n{res.stderr}")
        if verbose:
            sys.stderr.write(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_one, sources()))
    res = subprocess.run([nvcc, "-shared", "-cudart", "static", "-Xlinker", "-soname=libfstattn_b200.so", "-o", LIB, *objs], capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    _build_host()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
