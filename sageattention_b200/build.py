"""Builds libsage3_b200.so (sm_100a only, nvcc) and the host extension _host.so (g++, against the installed torch) next to this file.

Usage:  python -m sageattention_b200.build [--force]
The library is plain CUDA C++ behind a C ABI (include/sage3_b200.h); it links the CUDA runtime
statically and resolves the one driver entry point it needs at run time, so it has no link-time
dependency on libcuda or on PyTorch.
"""
from __future__ import annotations

import os
import pathlib
import subprocess
import sys

PKG = pathlib.Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libsage3_b200.so"
HOST_LIB = PKG / "_host.so"
HOST_SOURCE = "sage3_host.cpp"
SOURCES = ["sage3_abi.cu", "sage3_prepass.cu", "sage3_attn.cu"]
HEADERS = ["sage3_common.cuh", "sage3_kernels.h", "sage3_split.h"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]


def _stale() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    deps = [CSRC / s for s in SOURCES + HEADERS] + [PKG.parent / "include" / "sage3_b200.h", pathlib.Path(__file__)]
    return any(d.stat().st_mtime > t for d in deps)


def _build_host(force: bool) -> None:
    """The CPython extension behind the functional entry points (argument checks, output and workspace tensors)."""
    deps = [CSRC / HOST_SOURCE, PKG.parent / "include" / "sage3_b200.h", pathlib.Path(__file__)]
    if not force and HOST_LIB.exists() and all(d.stat().st_mtime <= HOST_LIB.stat().st_mtime for d in deps):
        return
    import sysconfig

    import torch
    root = pathlib.Path(torch.__file__).resolve().parent
    cuda = pathlib.Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    inc = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", cuda / "include", sysconfig.get_paths()["include"]]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-isystem{i}" for i in inc], str(CSRC / HOST_SOURCE),
           "-o", str(HOST_LIB), f"-L{root / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed on {HOST_SOURCE}:\n{r.stdout}")


def build(force: bool = False, verbose: bool = False) -> pathlib.Path:
    _build_host(force)
    if not force and not _stale():
        return LIB
    nvcc = os.environ.get("NVCC", "nvcc")
    objs = []
    procs = []
    obj_dir = PKG / "build"
    obj_dir.mkdir(exist_ok=True)
    for src in SOURCES:
        obj = obj_dir / (src + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(CSRC / src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(str(obj))
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
        if verbose:
            print(out)
    subprocess.check_call([nvcc, "-shared", "-o", str(LIB), *objs, "-Xcompiler", "-fvisibility=hidden"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
