"""The library's host code without a GPU: its object files linked with tests/fake_cudart.cpp, so that a call of the C ABI shows
which kernels it launches and what it does when a launch is refused."""
from __future__ import annotations

import ctypes
import functools
import os
import re
import shutil
import subprocess
import tempfile

from adkv_b200 import _lib, build

HERE = os.path.dirname(os.path.abspath(__file__))
PTR = 1 << 20        # any aligned address: nothing is launched, so nothing is read


@functools.lru_cache(None)
def library() -> ctypes.CDLL:
    objs = [os.path.join(build.OBJ_DIR, os.path.splitext(s)[0] + ".o") for s in build.SOURCES]
    deps = [os.path.join(build.CSRC, f) for f in build.SOURCES + build.HEADERS]
    if any(build._older(o, deps) for o in objs):
        build.build(force=True)
    out = os.path.join(tempfile.mkdtemp(prefix="adkv_fake_"), "libadkv_fake.so")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    subprocess.check_call([shutil.which("g++") or "g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I" + include,
                           os.path.join(HERE, "fake_cudart.cpp")] + objs + ["-o", out])
    lib = ctypes.CDLL(out)
    for name, argtypes in _lib.SIGNATURES.items():
        fn = getattr(lib, name)
        fn.argtypes, fn.restype = argtypes, _lib._RESTYPE.get(name, ctypes.c_int)
    lib.fake_launch.restype = ctypes.c_char_p
    return lib


def run(name, *args, fail=()):
    """Return code and launches ``(kernel, CTAs, threads, beside)`` of one call; ``fail``: runtime functions and which call of them fails."""
    lib = library()
    lib.fake_reset()
    for function, nth in fail:
        lib.fake_fail(function.encode(), nth)
    rc = getattr(lib, name)(*args)
    grid, block, beside = ctypes.c_uint(), ctypes.c_uint(), ctypes.c_int()
    out = []
    for i in range(lib.fake_launches()):
        kernel = lib.fake_launch(i, ctypes.byref(grid), ctypes.byref(block), ctypes.byref(beside)).decode()
        out.append((kernel, grid.value, block.value, bool(beside.value)))
    return rc, out


_params = _lib.Params(*[PTR] * 5)
_pp = ctypes.addressof(_params)


def prefill(B, H, T, bits=4, fail=()):
    ns = T // (32 // bits) + 1
    return run("adkv_encode_kv", PTR, PTR, _pp, PTR, PTR, PTR, _pp, PTR, B, H, T, 128, ns, bits, 0, 0.02, 50.0, None, fail=fail)


FAST = _lib.FLAG_FAST_REPLAY


def _step(name, *args, fail=()):
    """The decode kernel of one step, without ``decode_attn_`` and ``_kernel`` and its template arguments, and its CTAs; the return code
    and all launches where something is to fail."""
    rc, got = run(name, *args, fail=fail)
    if fail:
        return rc, got
    assert rc == 0, rc
    kernel = re.search(r"decode_attn_?(\w*?)_?kernelI", got[0][0]).group(1)
    return kernel or "whole", got[0][1]


def decode(bits, G, B, Hkv, T, bounds, tails=True, flags=FAST, fail=()):
    tail = PTR if tails else None
    return _step("adkv_decode_attn", PTR, PTR, PTR, PTR, PTR, _pp, _pp, tail, tail, None, 0, PTR, B, G * Hkv, Hkv, T, 128, T + 1, bits,
                 0.1, *bounds, flags, None, fail=fail)


def decode_varlen(bits, G, B, Hkv, room, bounds, flags=FAST):
    ns = -(-room // (32 // bits))
    return _step("adkv_decode_attn_varlen", PTR, PTR, PTR, PTR, PTR, _pp, _pp, PTR, PTR, PTR, PTR, B, G * Hkv, Hkv, 128, ns, bits, 0.1,
                 *bounds, flags, None)


def decode_ckpt(bits, G, B, Hkv, T, interval, bounds, flags=FAST, fail=()):
    return _step("adkv_decode_attn_ckpt", PTR, PTR, PTR, PTR, PTR, _pp, _pp, PTR, PTR, PTR, PTR, interval, T, None, 0, PTR, PTR, 1 << 40, B,
                 G * Hkv, Hkv, T, 128, T + 1, bits, 0.1, *bounds, flags, None, fail=fail)


def decode_static(bits, G, B, Hkv, T, interval, bounds, flags=FAST, fail=()):
    return _step("adkv_decode_attn_ckpt_static", PTR, PTR, PTR, PTR, PTR, _pp, _pp, PTR, PTR, PTR, PTR, interval, T, None, 0, PTR, B, G * Hkv, Hkv,
                 T, 128, T + 1, bits, 0.1, *bounds, flags, None, fail=fail)
