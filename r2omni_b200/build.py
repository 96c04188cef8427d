"""Build ``lib/libr2k_b200.so`` (nvcc for sm_100a) and ``lib/_r2k_host.so`` (the host module, a C++ torch extension) in-tree;
no GPU needed."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "lib", "libr2k_b200.so")
HOST_LIB = os.path.join(PKG, "lib", "_r2k_host.so")
HOST_TAG = os.path.join(PKG, "lib", "_r2k_host.tag")   # what the host module was built for
HOST_SOURCE = "host_ext.cpp"
SOURCES = ("r2k_api.cu",)
HEADERS = ("decode.cuh", "decode_consumer.cuh", "decode_kernel.cuh", "device_utils.cuh", "pack_kernels.cuh", "build_kernel.cuh")


def _stale(target: str, sources) -> bool:
    if not os.path.exists(target):
        return True
    built = os.path.getmtime(target)
    return any(os.path.getmtime(d) > built for d in sources)


def _host_tag() -> str:
    import torch

    return f"torch {torch.__version__}, {sys.implementation.cache_tag}"


def host_stale() -> bool:
    """Whether the host module is missing, older than its sources, or built for another torch or Python."""
    if _stale(HOST_LIB, (os.path.join(CSRC, HOST_SOURCE), os.path.join(ROOT, "include", "r2k_b200.h"))) or not os.path.exists(HOST_TAG):
        return True
    with open(HOST_TAG) as f:
        return f.read() != _host_tag()


def _build_host(force: bool) -> None:
    if not force and not host_stale():
        return
    import sysconfig

    import torch

    source = os.path.join(CSRC, HOST_SOURCE)
    torch_dir = os.path.dirname(torch.__file__)
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    includes = (os.path.join(ROOT, "include"), os.path.join(torch_dir, "include"),
                os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"), os.path.join(cuda_home, "include"),
                sysconfig.get_paths()["include"])
    cmd = ["g++", "-O3", "-std=c++17", "-shared", "-fPIC", "-DTORCH_EXTENSION_NAME=_r2k_host",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
    for path in includes:
        cmd += ["-isystem" if "torch" in path else "-I", path]
    cmd += ["-o", HOST_LIB, source, "-L", os.path.dirname(LIB), "-l:libr2k_b200.so", "-L", os.path.join(torch_dir, "lib"), "-ltorch_python",
            "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError("g++ failed:\n" + proc.stdout + proc.stderr)
    with open(HOST_TAG, "w") as f:
        f.write(_host_tag())


def build_library(force: bool = False, verbose: bool = False) -> str:
    sources = [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [os.path.join(ROOT, "include", "r2k_b200.h")]
    if not force and not _stale(LIB, sources):
        _build_host(force=False)
        return LIB
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build libr2k_b200.so")
    os.makedirs(os.path.dirname(LIB), exist_ok=True)
    cmd = [
        nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
        "-I", os.path.join(ROOT, "include"), "-I", CSRC, "--shared", "-Xcompiler", "-fPIC",
        "-o", LIB,
    ] + [os.path.join(CSRC, s) for s in SOURCES]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + proc.stdout + proc.stderr)
    if verbose:
        sys.stderr.write(proc.stderr)
    _build_host(force)
    return LIB


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
