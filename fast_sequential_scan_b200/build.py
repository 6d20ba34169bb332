"""In-tree build of ``libfss_b200.so`` (the C-ABI CUDA library) with plain nvcc for sm_100a, and of
``_fss_torch*.so`` (the autograd side of the entry points, ``csrc/fss_torch.cpp``) with g++ against torch.
The latter carries the Python and the torch it was compiled for in its name: one for another torch is neither
taken for up to date here nor loaded by the package.

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


def torch_lib() -> Path:
    """Where ``fss_torch.cpp`` is built for the running Python and torch."""
    import torch
    return PKG / f"_fss_torch.{sys.implementation.cache_tag}.torch-{torch.__version__}.so"


def build_torch(force: bool = False) -> Path:
    lib = torch_lib()
    inputs = [TORCH_SOURCE, PKG.parent / "include" / "fss_b200.h", Path(__file__)]
    if not force and lib.is_file() and lib.stat().st_mtime >= max(p.stat().st_mtime for p in inputs):
        return lib
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", Path(sysconfig.get_paths()["include"])]
    cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           "-DTORCH_EXTENSION_NAME=_fss_torch", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *[f"-I{p}" for p in includes], str(TORCH_SOURCE), "-o", str(lib), f"-L{root / 'lib'}",
           f"-Wl,-rpath,{root / 'lib'}", "-ltorch", "-ltorch_cpu", "-lc10", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError(f"g++ failed building {lib.name}")
    return lib


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
