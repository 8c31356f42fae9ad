"""Build ``libb200eagle.so`` (all CUDA kernels + the C ABI) in-tree with nvcc for sm_100a, and ``_b200ops.so`` (native
operator calls for Python, on top of that library and torch's C++ headers) with g++."""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libb200eagle.so")
OPS_SOURCE = os.path.join(CSRC, "ops.cpp")
OPS = os.path.join(HERE, "_b200ops.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall", "--threads", "0", "-shared",
]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def needs_build() -> bool:
    if not os.path.exists(LIB):
        return True
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + \
        glob.glob(os.path.join(ROOT, "include", "*.h"))
    return any(os.path.getmtime(d) > os.path.getmtime(LIB) for d in deps)


def build_ops(force: bool = False) -> str:
    """Compile the Python operator module against the library next to it (found there again at run time)."""
    import torch
    from torch.utils import cpp_extension
    header = os.path.join(ROOT, "include", "b200_eagle.h")
    if not force and os.path.exists(OPS) and all(os.path.getmtime(d) <= os.path.getmtime(OPS) for d in (OPS_SOURCE, header)):
        return OPS
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    includes = [os.path.join(ROOT, "include"), sysconfig.get_paths()["include"]] + cpp_extension.include_paths("cuda")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += [f for d in includes for f in ("-isystem", d)]
    cmd += ["-o", OPS, OPS_SOURCE, f"-L{torch_lib}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10_cuda", "-lc10",
            f"-L{HERE}", "-l:libb200eagle.so", "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{torch_lib}"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("g++ failed building _b200ops.so")
    return OPS


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every ``csrc/*.cu`` into one shared library, then the operator module; returns the library's path."""
    if not force and not needs_build():
        build_ops()
        return LIB
    nvcc = os.environ.get("NVCC", "nvcc")
    cmd = [nvcc] + NVCC_FLAGS + ["-I", os.path.join(ROOT, "include"), "-I", CSRC]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB] + sources()
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("nvcc failed building libb200eagle.so")
    if verbose:
        sys.stderr.write(res.stderr)
    build_ops(force=True)
    return LIB


if __name__ == "__main__":
    print(build(force=True, verbose="-v" in sys.argv))
