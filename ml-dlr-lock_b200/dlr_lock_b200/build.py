"""Build the C-ABI shared library in-tree with nvcc for sm_100a.

    python -m dlr_lock_b200.build        (or call build_library())

Every ``.cu`` under ``csrc/`` is compiled with
``-gencode arch=compute_100a,code=sm_100a -lineinfo`` and linked into
``libdlr_b200.so`` next to this file.  The CUDA runtime is linked statically,
so the library does not depend on which runtime the host process loaded.
``csrc/host.cpp`` becomes the Python module ``_host`` (walks over a net's
parameters; see there).
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

from . import _lib

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.normpath(os.path.join(HERE, "..", "csrc"))
INCLUDE = os.path.normpath(os.path.join(HERE, "..", "..", "include"))
LIB_PATH = os.path.join(HERE, "libdlr_b200.so")
HOST_SRC = os.path.join(CSRC, "host.cpp")
OBJ_DIR = os.path.join(HERE, "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--use_fast_math", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "-I", INCLUDE,
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the CUDA extension cannot be built")
    return exe


def _sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_host(force: bool = False) -> str:
    """Compile the host-side helper module ``_host`` against torch's headers, if there is none for this Python and torch or
    its source is newer."""
    path = _lib.host_path()
    if not force and not _stale(path, [HOST_SRC]):
        return path
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths

    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-I", sysconfig.get_paths()["include"]]
    for p in include_paths():
        cmd += ["-isystem", p]
    cmd += [HOST_SRC, "-o", path]
    for p in library_paths():
        cmd += ["-L", p]
    r = subprocess.run(cmd + ["-ltorch_python", "-ltorch_cpu", "-lc10"], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return path


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile what is out of date (the CUDA library and the host helper) and return the path of the shared library."""
    build_host(force)
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(INCLUDE, "dlr_b200.h"))
    nvcc = _nvcc()
    jobs = []
    objs = []
    for src in _sources():
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            jobs.append([nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj])

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stdout + r.stderr

    with ThreadPoolExecutor(max_workers=max(1, min(len(jobs), os.cpu_count() or 1))) as ex:
        for out in ex.map(run, jobs):
            if verbose and out:
                print(out)
    if jobs or force or _stale(LIB_PATH, objs):
        run([nvcc, "-shared", "-o", LIB_PATH] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"])
    return LIB_PATH


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
