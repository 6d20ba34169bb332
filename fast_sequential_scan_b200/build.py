"""In-tree build of ``libfss_b200.so`` (the C-ABI CUDA library) with plain nvcc for sm_100a, and of
``_fss_torch.so`` (the autograd side of the entry points, ``csrc/fss_torch.cpp``) with g++ against torch.

The library needs no libtorch and no pybind: its only inputs are ``csrc/*.cu[h]`` and
``include/fss_b200.h``.  The results sit beside this file so that they travel with the source tree.  Run as
``python fast_sequential_scan_b200/build.py`` (add ``--force`` to rebuild, ``--verbose`` for ptxas
resource usage); run it as a script, not with ``-m``: importing the package needs the library.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libfss_b200.so"
TORCH_SOURCE = CSRC / "fss_torch.cpp"
TORCH_LIB = PKG / "_fss_torch.so"

NVCC_FLAGS = [
    "-O3", "-std=c++17",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-Xcompiler", "-fPIC,-fvisibility=hidden",
    "-shared",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found: cannot build libfss_b200.so")
    return exe


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")) + [PKG.parent / "include" / "fss_b200.h"]


def is_stale() -> bool:
    if not LIB.is_file():
        return True
    t = LIB.stat().st_mtime
    return any(s.stat().st_mtime > t for s in sources() + [Path(__file__)])


def build_torch(force: bool = False) -> Path:
    inputs = [TORCH_SOURCE, PKG.parent / "include" / "fss_b200.h", Path(__file__)]
    if not force and TORCH_LIB.is_file() and TORCH_LIB.stat().st_mtime >= max(p.stat().st_mtime for p in inputs):
        return TORCH_LIB
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", Path(sysconfig.get_paths()["include"])]
    cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           "-DTORCH_EXTENSION_NAME=_fss_torch", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *[f"-I{p}" for p in includes], str(TORCH_SOURCE), "-o", str(TORCH_LIB), f"-L{root / 'lib'}",
           f"-Wl,-rpath,{root / 'lib'}", "-ltorch", "-ltorch_cpu", "-lc10", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("g++ failed building _fss_torch.so")
    return TORCH_LIB


def build(force: bool = False, verbose: bool = False) -> Path:
    build_torch(force)
    if not force and not is_stale():
        return LIB
    cmd = [_nvcc(), *NVCC_FLAGS]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", str(LIB)] + [str(f) for f in sorted(CSRC.glob("*.cu"))]
    env = dict(os.environ)
    res = subprocess.run(cmd, env=env, capture_output=True, text=True)
    if verbose or res.returncode:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode:
        raise RuntimeError("nvcc failed building libfss_b200.so")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
