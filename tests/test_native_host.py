"""The native host path of ``gemv.decode_attn``: what it takes over equals the Python path, what it does not take over is left
alone and refused or converted as before."""
import ctypes
import gc

import numpy as np
import pytest
import torch

from adkv_b200 import _lib, build, gemv, synth
from tests.util import SMAX, SMIN

B, H, D, T, BITS = 2, 2, 128, 40, 4


def _args(device, seed=0):
    g = torch.Generator().manual_seed(seed)
    kp, vp = (synth.gen_params(seed + i, H, D, BITS, device=device) for i in range(2))
    shape = (B, H, gemv.n_super_for(T + 1, BITS), D // 4, 4, 4)
    kc, vc = (torch.randint(0, 256, shape, dtype=torch.uint8, generator=g).to(device) for _ in range(2))
    q, kn, vn = (torch.randn(B, H, 1, D, generator=g).half().to(device) for _ in range(3))
    return [q, kc, vc, kn, vn, kp, vp, T, 0.1, SMIN, SMAX]


def _native(args, out=None, kt=None, vt=None, flags=0, bits=BITS):
    return _lib.host().decode(*args, bits, out, kt, vt, flags)


def test_host_memory_is_left_to_the_python_path():
    args = _args("cpu")
    assert _native(args) is None
    with pytest.raises(RuntimeError, match="k_cache must be a CUDA tensor"):
        gemv.decode_attn(*args)
    with pytest.raises(RuntimeError, match="q must be float16"):
        gemv.decode_attn(args[0].float(), *args[1:])


def _tails():
    return [torch.rand(B, H, 2, D, generator=torch.Generator().manual_seed(9)).cuda() + 0.1 for _ in range(2)]


@pytest.mark.gpu
@pytest.mark.parametrize("tails", [False, True])
@pytest.mark.parametrize("with_out", [False, True])
def test_equals_the_python_path(tails, with_out):
    res = []
    for native in (True, False):
        args = _args("cuda")
        kt, vt = _tails() if tails else (None, None)
        out = torch.empty(B, H, D, dtype=torch.float16, device="cuda") if with_out else None
        if not native:
            args[0] = args[0].as_subclass(type("T2", (torch.Tensor,), {}))      # a subclass is the Python path's business
        got = _native(args, out, kt, vt) if native else gemv.decode_attn(*args, bits=BITS, fast=False, out=out, k_tail=kt, v_tail=vt)
        assert isinstance(got, torch.Tensor) and (out is None or got is out)
        res.append([got, args[1], args[2]] + ([kt, vt] if tails else []))
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_what_the_native_path_leaves_alone():
    base, (kt, vt) = _args("cuda"), _tails()
    def other(i, x, **k):
        a = list(base)
        a[i] = x
        return _native(a, **k)
    strided = torch.empty(B, H, 2, D, dtype=torch.float16, device="cuda")[:, :, :1]
    before = base[1].clone()
    assert other(0, base[0].float()) is None and other(0, strided) is None and other(0, base[0][:1]) is None
    assert other(3, base[3][:, :1]) is None and other(4, strided) is None and other(0, torch.nn.Parameter(base[0]).cpu()) is None
    assert other(5, base[5][:4]) is None and other(6, tuple(t[:1] for t in base[6])) is None and other(5, iter(base[5])) is None
    assert other(7, -1) is None and other(7, 1 << 40) is None and other(7, float(T)) is None and other(7, np.int64(T)) is None
    assert other(7, base[1].shape[2] * 8) is None and other(8, 1) is None
    assert _native(base, bits=3) is None and _native(base, kt=kt) is None and _native(base, kt=kt, vt=vt[:1]) is None
    assert _native(base, kt=kt, vt=vt, flags=_lib.FLAG_HALF_STATE) is None
    assert _native(base, out=torch.empty(B, H, D, device="cuda")) is None
    assert torch.equal(base[1], before) and gemv.device_status() == 0
    got = gemv.decode_attn(strided.zero_(), *base[1:], bits=BITS)           # converted by the Python path, as before
    assert got.shape == (B, H, D)
    with pytest.raises(RuntimeError, match="group size"):                   # the library's refusals keep their text
        gemv.decode_attn(torch.zeros(B, 3 * H, 1, D, dtype=torch.float16, device="cuda"), *base[1:], bits=BITS)


@pytest.fixture
def no_host_module(monkeypatch):
    monkeypatch.setattr(build, "HOST_LIB", build.HOST_LIB + ".missing")
    monkeypatch.setattr(_lib, "_host", None)
    with pytest.warns(RuntimeWarning, match="argument checks stay in Python"):
        assert not _lib.host()


def test_without_the_host_module(no_host_module):
    """The Python path takes every call, its refusals included; only the first call says so."""
    args = _args("cpu")
    with pytest.raises(RuntimeError, match="k_cache must be a CUDA tensor"):
        gemv.decode_attn(*args)


def test_refusals_come_before_missing_kernels(monkeypatch):
    def missing():
        raise RuntimeError("libadkv_b200.so is missing")
    monkeypatch.setattr(_lib, "load", missing)
    monkeypatch.setattr(_lib, "_host", None)
    with pytest.raises(RuntimeError, match="q must be float16"):
        args = _args("cpu")
        gemv.decode_attn(args[0].float(), *args[1:])


def test_build_goes_on_without_the_host_module(monkeypatch, tmp_path, capsys):
    """A torch of another version or Python asks for another file; a compiler that is missing costs the host module only."""
    assert torch.__version__ in build.HOST_LIB and build.HOST_LIB.endswith(".so")
    monkeypatch.setattr(build, "HOST_LIB", str(tmp_path / "other_torch.so"))
    monkeypatch.setattr(build, "HOST_SOURCE", str(tmp_path / "missing.cpp"))
    monkeypatch.setattr(build, "is_stale", lambda: False)
    monkeypatch.setattr(build, "host_is_stale", lambda: True)
    assert build.build() == build.LIB
    assert "host module not built" in capsys.readouterr().err


@pytest.mark.gpu
def test_results_without_the_host_module(request):
    want = gemv.decode_attn(*_args("cuda"), bits=BITS)
    request.getfixturevalue("no_host_module")
    assert torch.equal(gemv.decode_attn(*_args("cuda"), bits=BITS), want)


def _step(native, Hq=H, out=None, **kw):
    args = _args("cuda")
    args[0] = torch.randn(B, Hq, 1, D, generator=torch.Generator().manual_seed(5)).half().cuda().requires_grad_()
    kt, vt = (None, None) if kw.get("half_state") else _tails()
    q = args[0] if native else args[0].as_subclass(type("T2", (torch.Tensor,), {}))
    got = gemv.decode_attn(q, *args[1:], bits=BITS, out=out, k_tail=kt, v_tail=vt, **kw)
    assert not got.requires_grad
    return [got, args[1], args[2]] + ([] if kt is None else [kt, vt])


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(Hq=4 * H), dict(half_state=True), dict(tail_keep=True), dict(split_channels=True, fast=False)])
def test_options_equal_the_python_path(kw):
    for a, b in zip(_step(True, **kw), _step(False, **kw)):
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_side_stream_and_capture():
    """The native path launches on the current stream: a side stream sees its own inputs, a capture records the step."""
    want = _step(False, tail_keep=True)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        got = _step(True, tail_keep=True)
        args, (kt, vt) = _args("cuda"), _tails()
    s.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    ref = gemv.decode_attn(*args, bits=BITS, k_tail=kt, v_tail=vt, tail_keep=True).clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = gemv.decode_attn(*args, bits=BITS, k_tail=kt, v_tail=vt, tail_keep=True)
    out.zero_()
    graph.replay()
    assert torch.equal(out, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("rc", [0, -3])
def test_one_launch_a_step(rc):
    """Nothing that may fail is left to be done once the step is launched (the Python path would launch it again): the result's
    Python object is there when the library is called."""
    seen = []

    @ctypes.CFUNCTYPE(ctypes.c_int, *_lib.SIGNATURES["adkv_decode_attn"])
    def launch(*a):
        seen.append(any(type(o) is torch.Tensor and o.is_cuda and o.data_ptr() == a[11] for o in gc.get_objects()))
        return rc

    args = _args("cuda")
    host = _lib.host()
    host.bind(ctypes.cast(launch, ctypes.c_void_p).value)
    try:
        if rc:
            with pytest.raises(RuntimeError, match="decode_attn"):
                gemv.decode_attn(*args, bits=BITS)
        else:
            assert gemv.decode_attn(*args, bits=BITS).shape == (B, H, D)
    finally:
        host.bind(ctypes.cast(_lib.load().adkv_decode_attn, ctypes.c_void_p).value)
    assert seen == [True]
