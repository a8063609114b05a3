"""Builds ``lib/libb200q.so`` from ``csrc/*.cu`` with nvcc for sm_100a, and the extension module ``lib/_b200q_host.so``
(the operators' native call path, ``csrc/host_ops.cpp``) with the host compiler.

    python build.py            # from this directory, or
    build.build()              # from Python

nvcc cross-compiles without a GPU.  Objects are cached under ``build/`` and rebuilt when a
source or header is newer.  The library has a plain C ABI (include/b200q.h at the repository
root) and no dependency on Python or torch.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
OBJ = HERE / "build"
LIB = HERE / "lib" / "libb200q.so"
HOST_SRC = CSRC / "host_ops.cpp"
HOST_LIB = HERE / "lib" / "_b200q_host.so"
HEADER = HERE.parent / "include" / "b200q.h"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build libb200q.so")
    return exe


def _newer(target: Path, deps) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def _build_host(verbose: bool, force: bool) -> None:
    """The call path needs the headers and libraries of the installed torch; the CUDA library does not."""
    if not force and not _newer(HOST_LIB, [HOST_SRC]):
        return
    import torch
    root = Path(torch.__file__).resolve().parent
    cuda_include = Path(_nvcc()).resolve().parents[1] / "include"
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-isystem{d}" for d in (sysconfig.get_paths()["include"], root / "include",
                                      root / "include" / "torch" / "csrc" / "api" / "include", cuda_include)),
           str(HOST_SRC), "-o", str(HOST_LIB), f"-L{root / 'lib'}", f"-Wl,-rpath,{root / 'lib'}",
           "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10_cuda", "-lc10"]
    if verbose:
        print(" ".join(cmd), flush=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed for {HOST_SRC.name}:\n{res.stdout}\n{res.stderr}")


def build(verbose: bool = False, force: bool = False) -> Path:
    sources = sorted(CSRC.glob("*.cu"))
    headers = sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h")) + [HEADER]
    OBJ.mkdir(exist_ok=True)
    LIB.parent.mkdir(exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: Path):
        obj = OBJ / (src.stem + ".o")
        if force or _newer(obj, [src, *headers]):
            cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
            if verbose:
                print(" ".join(cmd), flush=True)
            res = subprocess.run(cmd, capture_output=True, text=True)
            if res.returncode != 0:
                raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        host = pool.submit(_build_host, verbose, force)
        objs = list(pool.map(compile_one, sources))
        host.result()
    if force or _newer(LIB, objs):
        cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a"]
        if verbose:
            print(" ".join(cmd), flush=True)
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(verbose=True, force="--force" in sys.argv))
