"""Builds the two native parts of this package in-tree.

    python -m triton_sigmoid_b200.build [--force] [--verbose]

``triton_sigmoid_b200/lib/libsigattn_b200.so`` (nvcc, sm_100a only) exports the C ABI declared in
``include/sigattn_b200.h``; nvcc cross-compiles without a GPU.
``triton_sigmoid_b200/lib/_sigattn_torch.so`` (g++) is the eager host path between torch and that ABI.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

from ._paths import CSRC, EXT_PATH, LIB_DIR, LIB_PATH, PKG_DIR, ROOT  # noqa: F401

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
]


EXT_SOURCE = os.path.join(CSRC, "torch_ext.cpp")
HEADER = os.path.join(ROOT, "include", "sigattn_b200.h")


def _sources():
    srcs = [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))]
    srcs.append(HEADER)
    return srcs


def _stale(target, sources) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(s) > t for s in sources)


def needs_build() -> bool:
    return _stale(LIB_PATH, _sources()) or _stale(EXT_PATH, [EXT_SOURCE, HEADER])


def find_nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: set NVCC or put it on PATH")


def _run(cmd, target, verbose):
    os.makedirs(os.path.dirname(target), exist_ok=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed building {target}")


def build_ext(force: bool = False, verbose: bool = False) -> str:
    """Compile the torch extension (host code only)."""
    if not force and not _stale(EXT_PATH, [EXT_SOURCE, HEADER]):
        return EXT_PATH
    import torch

    root = torch.__path__[0]
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(find_nvcc())))
    includes = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    # the system's g++ (which nvcc uses as well), not $CXX: a compiler that links its own static libstdc++ into the
    # extension gives it a second copy of the iostream and locale state that torch's error formatting relies on
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{d}" for d in includes), EXT_SOURCE,
           "-o", EXT_PATH, f"-L{os.path.join(root, 'lib')}", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python",
           "-lc10", "-lc10_cuda"]
    _run(cmd, EXT_PATH, verbose)
    return EXT_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the library and the torch extension (each skipped when newer than its sources, unless `force`)."""
    if force or _stale(LIB_PATH, _sources()):
        cmd = [find_nvcc(), *NVCC_FLAGS]
        if verbose:
            cmd += ["-Xptxas", "-v"]
        cmd += ["-o", LIB_PATH, os.path.join(CSRC, "sigattn_api.cu")]
        _run(cmd, LIB_PATH, verbose)
    build_ext(force, verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
