"""Builds ``liboeq_b200.so`` (the C-ABI runtime) in-tree with nvcc for sm_100a, and ``liboeq_torch.so`` (the torch
library ops on top of it) with the host compiler.

The library holds the host runtime and the fixed kernels; the problem-specific
kernels are specialised at run time from ``csrc/*.cuh`` and cached under
``_kcache/``.  ``python -m openequivariance_b200.build`` rebuilds the library.
"""

from __future__ import annotations

import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "liboeq_b200.so")
SOURCES = ["oeq_runtime.cu"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; the CUDA toolkit is required to build liboeq_b200.so")


def _stale(target: str, deps) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(d) > os.path.getmtime(target) for d in deps)


def _build(target: str, deps, command, verbose: bool, force: bool) -> str:
    """Run ``command(output)`` if ``target`` is missing or older than its sources.

    Several processes may get here at once (one rank per GPU under ``torch.distributed.run``): the build
    runs under an exclusive lock on a sidecar file, writes to a temporary name and is renamed into place,
    so no process ever loads a half-written library; whoever waited for the lock re-checks and usually
    finds the work done.
    """
    if not force and not _stale(target, deps):
        return target
    import fcntl
    with open(target + ".lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if not force and not _stale(target, deps):
                return target
            tmp = f"{target}.tmp{os.getpid()}"
            cmd = command(tmp)
            res = subprocess.run(cmd, capture_output=True, text=True)
            if res.returncode != 0:
                if os.path.exists(tmp):
                    os.remove(tmp)
                raise RuntimeError(f"building {os.path.basename(target)} failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
            os.replace(tmp, target)
            if verbose:
                print(res.stdout + res.stderr)
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)
    return target


HEADER = os.path.join(HERE, "..", "include", "oeq_b200.h")


def build_library(force: bool = False, verbose: bool = False) -> str:
    """The C-ABI runtime."""
    sources = [os.path.join(CSRC, s) for s in SOURCES]

    def command(out):
        cmd = [_nvcc(), "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-lineinfo",
               "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static", "-o", out] + sources + ["-ldl"]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        if os.environ.get("OEQ_DEV_PROFILE"):
            cmd.insert(1, "-DOEQ_DEV_PROFILE")      # development build: cycle accounting inside the kernels
        return cmd

    return _build(LIB, sources + [HEADER], command, verbose, force)


def torch_library_path() -> str:
    """One file per torch release: the library uses its C++ interface."""
    import torch
    return os.path.join(HERE, f"liboeq_torch-{torch.__version__.split('+')[0]}.so")


def build_torch_library(force: bool = False, verbose: bool = False) -> str:
    """The torch library ops; links against the runtime beside it and the installed torch."""
    import torch
    lib = build_library(verbose=verbose)
    root = os.path.dirname(torch.__file__)
    include = os.path.join(root, "include")
    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    source = os.path.join(CSRC, "oeq_torch.cpp")

    # The host compiler that nvcc uses, not $CXX: the library hands C++ objects to and from torch and has to share its
    # libstdc++.  With a second copy linked in, the first number written to a stream (an error message) ends the process.
    def command(out):
        return ["g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-I" + include,
                "-I" + os.path.join(include, "torch", "csrc", "api", "include"), "-I" + cuda, source, "-o", out,
                "-L" + os.path.join(root, "lib"), "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda",
                "-L" + HERE, "-l:" + os.path.basename(lib), "-Wl,-rpath,$ORIGIN"]

    return _build(torch_library_path(), [source, HEADER, os.path.abspath(__file__)], command, verbose, force)


if __name__ == "__main__":
    print(build_library(force=True, verbose=True))
    print(build_torch_library(force=True, verbose=True))
