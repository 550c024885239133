"""Builds the two native parts of the package in-tree.

    python -m mamba_b200.build          # or: from mamba_b200.build import build_library

libmamba_b200.so: the C-ABI library with the kernels; every .cu under csrc/ is compiled for sm_100a only.
nvcc cross-compiles without a GPU, so the build also runs on a CPU-only box.
_mamba_b200_host.so: the Python extension with the host side of the calls (csrc/host/*.cpp: checks, allocations,
autograd nodes, launches), compiled against the installed torch and linked to the library above.
"""
from __future__ import annotations

import os
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
OBJDIR = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libmamba_b200.so")
HOST_SRC = os.path.join(CSRC, "host")
HOST_LIB = os.path.join(HERE, "_mamba_b200_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++20",
    "-Xcompiler", "-fPIC", "-I", INCLUDE, "-I", CSRC,
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build libmamba_b200.so")
    return exe


def _host_flags():
    """Compiler flags for the extension: torch's, Python's and CUDA's headers."""
    import sysconfig
    import torch
    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    dirs = [INCLUDE, HOST_SRC, inc, os.path.join(inc, "torch", "csrc", "api", "include"), os.path.join(cuda, "include"),
            sysconfig.get_paths()["include"]]
    return ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_mamba_b200_host",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + [f for d in dirs for f in ("-isystem", d)]


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile whatever is out of date (both libraries) and return the path of libmamba_b200.so."""
    nvcc = _nvcc()
    os.makedirs(OBJDIR, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(INCLUDE, "mamba_b200.h"))
    jobs, objs, host_objs = [], [], []
    for src in _sources():
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJDIR, src[:-3] + ".o")
        objs.append(o)
        if force or _stale(o, [s] + headers):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            jobs.append(cmd)

    host_headers = [os.path.join(HOST_SRC, f) for f in os.listdir(HOST_SRC) if f.endswith(".h")]
    host_headers.append(os.path.join(INCLUDE, "mamba_b200.h"))
    host_flags = None
    for src in sorted(f for f in os.listdir(HOST_SRC) if f.endswith(".cpp")):
        s, o = os.path.join(HOST_SRC, src), os.path.join(OBJDIR, "host_" + src[:-4] + ".o")
        host_objs.append(o)
        if force or _stale(o, [s] + host_headers):
            host_flags = host_flags or _host_flags()
            jobs.append(["g++"] + host_flags + ["-c", s, "-o", o])

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(cmd[0] + " failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    if jobs:
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for log in ex.map(run, jobs):
                if verbose and log:
                    print(log)
    if force or jobs or _stale(LIB, objs):
        run([nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"])
    if force or jobs or _stale(HOST_LIB, host_objs + [LIB]):
        import torch
        torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
        cuda_lib = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "lib64")
        run(["g++", "-shared", "-o", HOST_LIB] + host_objs + [LIB, "-L" + torch_lib, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
             "-ltorch", "-ltorch_python", "-L" + cuda_lib, "-lcudart", "-Wl,-rpath,$ORIGIN", "-Wl,--no-as-needed"])
    return LIB


if __name__ == "__main__":
    import sys
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
