"""Build libawq_b200.so in-tree with nvcc for sm_100a (no GPU needed to compile), and the native
host path _native.so (csrc/host_ops.cpp) against the installed torch.

    python server-benchmark_b200/build.py [--force] [--verbose]

Both land next to the Python host code (awq_b200/) so that they travel with the source tree.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "awq_b200", "libawq_b200.so")
NATIVE_SRC = os.path.join(CSRC, "host_ops.cpp")
NATIVE_OUT = os.path.join(HERE, "awq_b200", "_native.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared",
    "-cudart", "static",
]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale(out: str, deps: list[str]) -> bool:
    if not os.path.exists(out):
        return True
    t = os.path.getmtime(out)
    return any(os.path.getmtime(d) > t for d in deps)


def _headers() -> list[str]:
    return glob.glob(os.path.join(HERE, "..", "include", "*.h"))


def _run(cmd: list[str], out: str, verbose: bool) -> None:
    res = subprocess.run([*cmd, "-o", out + ".tmp"], capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed building {os.path.basename(out)}")
    os.replace(out + ".tmp", out)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into one shared library, then the host path that links to
    it; returns the library's path."""
    if force or _stale(OUT, sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + _headers()):
        nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
        if not os.path.exists(nvcc):
            raise RuntimeError("nvcc not found: cannot build libawq_b200.so")
        _run([nvcc, *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), *sources()], OUT, verbose)
    if force or _stale(NATIVE_OUT, [NATIVE_SRC] + _headers()):
        _build_native(verbose)
    return OUT


def _build_native(verbose: bool) -> None:
    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I" + os.path.join(root, "include"),
           "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(cuda, "include"),
           NATIVE_SRC, "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cuda",
           "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10",
           "-L" + os.path.dirname(OUT), "-l:libawq_b200.so", "-Wl,-rpath,$ORIGIN"]
    _run(cmd, NATIVE_OUT, verbose)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
