"""Build libmegabake_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU), and beside it the small
library that puts the two ops' common case under PyTorch's dispatcher.

    python -m megabake_b200.build [--force]
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PACKAGE = Path(__file__).resolve().parent
CSRC = PACKAGE / "csrc"
LIBRARY = PACKAGE / "libmegabake_b200.so"
SOURCES = sorted(CSRC.glob("*.cu"))
OPS_SOURCE = CSRC / "torch_ops.cpp"


def ops_library() -> Path:
    """The ops' C++ registration is built against one PyTorch, and its name says which: another one's is not there."""
    import torch

    return PACKAGE / f"libmegabake_b200_ops-torch{torch.__version__}.so"


def headers() -> list[Path]:
    """Every header the library is built from: a new .cuh cannot be forgotten."""
    return sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h")) + sorted((PACKAGE.parent / "include").glob("*.h"))


NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--threads", "0", "-shared", "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build megabake_b200")
    return nvcc


def is_stale() -> bool:
    if not LIBRARY.exists():
        return True
    built = LIBRARY.stat().st_mtime
    return any(path.stat().st_mtime > built for path in SOURCES + headers())


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile the CUDA library if it is missing or older than its sources."""
    if not force and not is_stale():
        return LIBRARY
    command = [find_nvcc(), *NVCC_FLAGS, "-o", str(LIBRARY), *map(str, SOURCES), "-lcudart"]
    result = subprocess.run(command, capture_output=True, text=True)
    if verbose or result.returncode:
        sys.stderr.write(result.stdout + result.stderr)
    if result.returncode:
        raise RuntimeError(f"nvcc failed with exit code {result.returncode}")
    (PACKAGE / "build_log.txt").write_text(result.stdout + result.stderr)
    return LIBRARY


def build_ops(force: bool = False, verbose: bool = False) -> Path:
    """Compile the ops' C++ registration against the installed PyTorch if there is none for it or it is older than its sources."""
    library = ops_library()
    sources = [OPS_SOURCE, PACKAGE.parent / "include" / "megabake_b200.h"]
    if not force and library.exists() and all(path.stat().st_mtime <= library.stat().st_mtime for path in sources):
        return library
    import torch
    from torch.utils import cpp_extension

    command = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", "-o", str(library), str(OPS_SOURCE),
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
               *(f"-isystem{path}" for path in cpp_extension.include_paths(device_type="cuda")),
               *(f"-L{path}" for path in cpp_extension.library_paths(device_type="cuda")), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-lcudart"]
    result = subprocess.run(command, capture_output=True, text=True)
    if verbose or result.returncode:
        sys.stderr.write(result.stdout + result.stderr)
    if result.returncode:
        raise RuntimeError(f"{command[0]} failed with exit code {result.returncode}")
    return library


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
    print(build_ops(force="--force" in sys.argv, verbose=True))
