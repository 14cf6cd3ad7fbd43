"""Builds libnvllm_b200.so (the C-ABI library) in-tree with nvcc for sm_100a, and _host.so (the
CPython extension that holds the entry points' host path) with g++ against torch's headers.

Run as ``python -m nano_vllm_b200.build``.  nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_PATH = PKG_DIR / "libnvllm_b200.so"
HOST_PATH = PKG_DIR / "_host.so"
HOST_SOURCE = CSRC / "host.cpp"
HEADER = PKG_DIR.parent / "include" / "nvllm_b200.h"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--use_fast_math",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden",
    "-shared",
    "-cudart", "static",
]


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; the CUDA library cannot be built")


def _older(target: Path, deps) -> bool:
    return not target.exists() or any(d.stat().st_mtime > target.stat().st_mtime for d in deps)


def is_stale() -> bool:
    return _older(LIB_PATH, [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), HEADER]) or _older(HOST_PATH, [HOST_SOURCE, HEADER])


def _run(cmd: list[str], target: Path) -> str:
    """Runs a compiler that writes to a private name, then renames: a process that loads the library
    while another one builds it sees either the old file or the complete new one."""
    tmp = target.with_name(f".{target.name}.{os.getpid()}.tmp")
    cmd = [*cmd, "-o", str(tmp)]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        tmp.unlink(missing_ok=True)
        raise RuntimeError(f"{cmd[0]} failed:\n" + " ".join(cmd) + "\n" + proc.stdout + proc.stderr)
    os.replace(tmp, target)
    return proc.stderr


def _host_command() -> list[str]:
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", cuda / "include",
                Path(sysconfig.get_path("include"))]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-isystem{p}" for p in includes),
            str(HOST_SOURCE), f"-L{root / 'lib'}", f"-L{cuda / 'lib64'}", "-ltorch_python", "-ltorch", "-ltorch_cpu",
            "-lc10_cuda", "-lc10", "-l:libcudart.so.12", "-ldl"]


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compiles every .cu under csrc/ into one shared library and host.cpp into the extension module;
    returns the library's path."""
    if force or _older(HOST_PATH, [HOST_SOURCE, HEADER]):
        _run(_host_command(), HOST_PATH)
    if force or _older(LIB_PATH, [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), HEADER]):
        log = _run([_nvcc(), *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), *map(str, sources())], LIB_PATH)
        if verbose:
            sys.stderr.write(log)
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
