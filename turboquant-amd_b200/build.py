#!/usr/bin/env python3
"""Build libtq_b200.so (the C-ABI launcher library) for sm_100a with nvcc, and _tq_host.so (the host path) with g++.

    python turboquant-amd_b200/build.py [--verbose]

Objects go to turboquant-amd_b200/build/, the libraries to
turboquant-amd_b200/turboquant/lib/ (git-ignored).  nvcc
cross-compiles, so this works on a machine without a GPU.
"""
from __future__ import annotations

import importlib.util
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "turboquant", "lib", "libtq_b200.so")
HOST_LIB = os.path.join(HERE, "turboquant", "lib", "_tq_host.so")
SOURCES = ["tq_compress.cu", "tq_decode.cu", "tq_packed_attention.cu"]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a",
         "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_host() -> str:
    """The CPython extension against torch's C++ headers; torch's libraries are loaded before it, so no run path."""
    src = os.path.join(CSRC, "tq_host.cpp")
    if _stale(HOST_LIB, [src, os.path.join(HERE, "..", "include", "tq_b200.h"), os.path.abspath(__file__)]):
        torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
        include = os.path.join(torch_dir, "include")
        cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-I{include}",
               f"-I{os.path.join(include, 'torch', 'csrc', 'api', 'include')}",
               f"-I{os.path.join(os.path.dirname(os.path.dirname(NVCC)), 'include')}",
               f"-I{sysconfig.get_paths()['include']}", src, "-o", HOST_LIB, f"-L{os.path.join(torch_dir, 'lib')}",
               "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-ldl"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"g++ failed on tq_host.cpp:\n{res.stdout}\n{res.stderr}")
    return HOST_LIB


def build(verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    os.makedirs(os.path.dirname(LIB), exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".inc"))]
    headers.append(os.path.join(HERE, "..", "include", "tq_b200.h"))
    headers.append(os.path.abspath(__file__))

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ, src.replace(".cu", ".o"))
        path = os.path.join(CSRC, src)
        if _stale(obj, [path, *headers]):
            res = subprocess.run([NVCC, *FLAGS, "-c", path, "-o", obj], capture_output=True, text=True)
            with open(obj + ".log", "w") as fh:
                fh.write(res.stdout + res.stderr)
            if res.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src}:\n{res.stdout}\n{res.stderr}")
            if verbose:
                print(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES) + 1) as pool:
        host = pool.submit(build_host)
        objs = list(pool.map(compile_one, SOURCES))
        host.result()
    if _stale(LIB, objs):
        res = subprocess.run([NVCC, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"],
                             capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(verbose="--verbose" in sys.argv))
