"""Build the native parts in-tree: libgla_b200.so (nvcc, sm_100a) and _front.so (its PyTorch face, g++).

    python -m gtr_b200.build [--force] [-v]
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
SRC_DIR = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(ROOT, "include")
SOURCES = [os.path.join(SRC_DIR, "gla_b200.cu")]
HEADERS = [os.path.join(SRC_DIR, name) for name in
           ("gla_kernel.cuh", "gla_block.cuh", "gla_tiles.cuh", "gla_device.cuh", "gla_cluster.cuh", "gla_step.cuh", "swiglu_dwconv.cuh", "gla_bwd.cuh")]
HEADERS.append(os.path.join(INCLUDE, "gla_b200.h"))
OUT = os.path.join(PKG, "libgla_b200.so")
FRONT_SOURCES = [os.path.join(SRC_DIR, "torch_front.cpp")]
FRONT_HEADERS = [os.path.join(INCLUDE, "gla_b200.h")]
FRONT_OUT = os.path.join(PKG, "_front.so")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-shared", "-Xcompiler", "-fPIC", "-I", INCLUDE]


def nvcc() -> str:
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def front_command() -> list:
    import torch
    torch_dir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(nvcc())) or "/usr/local/cuda"
    includes = [INCLUDE, os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    lib = os.path.join(torch_dir, "lib")
    return ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-w",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *(f"-I{p}" for p in includes), *FRONT_SOURCES, "-o", FRONT_OUT, f"-L{lib}", f"-Wl,-rpath,{lib}",
            "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]


def up_to_date(out: str, inputs: list) -> bool:
    return os.path.exists(out) and all(os.path.getmtime(p) <= os.path.getmtime(out) for p in inputs)


def _run(cmd: list) -> str:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed:\n{' '.join(cmd)}\n{proc.stdout}\n{proc.stderr}")
    return proc.stderr


def build(force: bool = False, verbose: bool = False) -> str:
    if force or not up_to_date(FRONT_OUT, FRONT_SOURCES + FRONT_HEADERS):
        _run(front_command())
    if force or not up_to_date(OUT, SOURCES + HEADERS):
        log = _run([nvcc(), *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-o", OUT, *SOURCES])
        if verbose:
            print(log)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
