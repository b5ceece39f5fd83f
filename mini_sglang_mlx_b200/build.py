"""In-tree build of the C-ABI library ``libmsgl_b200.so`` (sm_100a only) and of the host module
``_host.so`` that calls it.

``python -m mini_sglang_mlx_b200.build`` compiles ``csrc/abi.cu`` (which
includes every kernel header) with nvcc into the package directory, so the
shared object travels with the source tree.  nvcc cross-compiles without a
GPU.  ``csrc/host_ops.cpp`` (tensor checks, scratch, launches on behalf of the Python operators) is
compiled with g++ against torch's headers and links the library by ``$ORIGIN``.  A rebuild happens
only when a source file is newer than what it makes.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
INCLUDE = PKG_DIR.parent / "include"
LIB_PATH = PKG_DIR / "libmsgl_b200.so"
HOST_PATH = PKG_DIR / "_host.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--shared", "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
]


def _stale(target: Path, sources: list[Path]) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(s.stat().st_mtime > t for s in sources)


def _library_sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")) + sorted(INCLUDE.glob("*.h"))


def _host_sources() -> list[Path]:
    return [CSRC / "host_ops.cpp"] + sorted(INCLUDE.glob("*.h"))


def needs_build() -> bool:
    return _stale(LIB_PATH, _library_sources()) or _stale(HOST_PATH, _host_sources())


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build libmsgl_b200.so")
    return nvcc


def _run(cmd: list[str], target: Path, verbose: bool) -> None:
    """Compile into a temporary name, then put the result in place in one step."""
    tmp = target.with_suffix(".so.tmp")
    proc = subprocess.run([*cmd, "-o", str(tmp)], capture_output=True, text=True)
    if verbose or proc.returncode != 0:
        sys.stderr.write(proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed with exit code {proc.returncode}")
    os.replace(tmp, target)


def _host_command() -> list[str]:
    import torch

    root = Path(torch.__file__).resolve().parent
    nvcc_root = Path(find_nvcc()).resolve().parent.parent
    inc = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include",
           nvcc_root / "include", Path(sysconfig.get_paths()["include"]), INCLUDE]
    return [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *[f"-I{p}" for p in inc], str(CSRC / "host_ops.cpp"), f"-L{root / 'lib'}", "-lc10", "-lc10_cuda",
            "-ltorch_cpu", "-ltorch_python", f"-L{PKG_DIR}", "-l:libmsgl_b200.so", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile what is missing or stale; return the path of the C-ABI library."""
    if force or _stale(LIB_PATH, _library_sources()):
        cus = [str(p) for p in sorted(CSRC.glob("*.cu"))]
        _run([find_nvcc(), *NVCC_FLAGS, f"-I{INCLUDE}", *cus], LIB_PATH, verbose)
    if force or _stale(HOST_PATH, _host_sources()):
        _run(_host_command(), HOST_PATH, verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
