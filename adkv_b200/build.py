"""Build the C-ABI shared library ``adkv_b200/lib/libadkv_b200.so`` for sm_100a with nvcc, and the host module of gemv.py.

The library has no dependency on torch or Python: plain ``extern "C"`` entry points declared in
``include/adkv_b200.h``.  The host module checks torch tensors and calls it; it is bound to the torch and Python it was built
with, which its file name says, and ``gemv.py`` does without it where it is missing.  Both are built in-tree so that they
travel with the source snapshot.
"""
from __future__ import annotations

import importlib.metadata
import os
import shutil
from concurrent.futures import ThreadPoolExecutor
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB = os.path.join(LIB_DIR, "libadkv_b200.so")

def _host_lib() -> str | None:
    """Argument checks of gemv.decode_attn, compiled against the headers of the installed torch (None without one)."""
    try:
        torch_version = importlib.metadata.version("torch")
    except importlib.metadata.PackageNotFoundError:
        return None
    return os.path.join(LIB_DIR, f"_adkv_pyhost-torch{torch_version}{sysconfig.get_config_var('EXT_SUFFIX')}")


HOST_LIB = _host_lib()
HOST_SOURCE = os.path.join(CSRC, "adkv_pyhost.cpp")
SOURCES = ["adkv_capi.cu", "adkv_encode.cu", "adkv_fused.cu", "adkv_unfused.cu", "adkv_split.cu", "adkv_wide.cu",
           "adkv_half.cu", "adkv_narrow.cu", "adkv_segments.cu", "adkv_tensor.cu"]
HEADERS = ["adkv_device.cuh", "adkv_decode.cuh", "adkv_softmax.cuh", "adkv_half.cuh", "adkv_io.cuh", "adkv_host.h",
           "adkv_narrow.cuh", "adkv_tensor.cuh",
           os.path.join("..", "..", "include", "adkv_b200.h")]
OBJ_DIR = os.path.join(PKG, "build")

NVCC_FLAGS = ["-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
              "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the CUDA toolkit is required to build libadkv_b200.so")
    return exe


def _older(path: str, deps: list[str]) -> bool:
    return not os.path.exists(path) or any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps)


def is_stale() -> bool:
    return _older(LIB, [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [os.path.abspath(__file__)])


def host_is_stale() -> bool:
    header = os.path.join(CSRC, HEADERS[-1])
    return HOST_LIB is not None and _older(HOST_LIB, [HOST_SOURCE, header, os.path.abspath(__file__)])


def build_host(verbose: bool = False) -> str:
    import torch
    torch_dir = os.path.dirname(os.path.abspath(torch.__file__))
    inc = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")]
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", HOST_SOURCE, "-o", HOST_LIB]
    cmd += ["-I" + d for d in inc] + ["-L" + os.path.join(torch_dir, "lib")]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.check_call(cmd)
    return HOST_LIB


def build(force: bool = False, verbose: bool = False, extra: list[str] | None = None) -> str:
    if force or is_stale():
        _build_library(verbose, extra)
    if HOST_LIB is not None and (force or host_is_stale()):
        try:
            build_host(verbose)
        except (ImportError, OSError, subprocess.CalledProcessError) as e:   # the library does not need it
            print(f"host module not built, gemv.decode_attn checks its arguments in Python: {e}", file=sys.stderr)
    return LIB


def _build_library(verbose: bool, extra: list[str] | None) -> None:
    os.makedirs(LIB_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ_DIR, os.path.splitext(src)[0] + ".o")
        cmd = [nvcc] + NVCC_FLAGS + (extra or []) + ["-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.check_call(cmd)
        return obj

    # the translation units are independent: compile them side by side, then link
    with ThreadPoolExecutor(max_workers=len(SOURCES)) as pool:
        objs = list(pool.map(compile_one, SOURCES))
    link = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a"] + objs + ["-o", LIB]
    if verbose:
        print(" ".join(link), flush=True)
    subprocess.check_call(link)


if __name__ == "__main__":
    build(force=True, verbose=True, extra=["-Xptxas", "-v"] if "-v" in sys.argv else None)
