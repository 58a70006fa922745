"""Decode steps on the tensor cores (next to tail states, up to four query heads per KV head) against the oracle and the
one-warp-per-tensor scan.  Sizes are the edges of the 64-token tiles and of the 16 tokens that a product of V takes, scales
at and outside the clamp bounds, values near the ends of fp16, more streams than a round of the chip holds.  Needs a B200."""
import ctypes
import time

import numpy as np
import pytest
import torch

from adkv_b200 import _lib, gemv
from oracle import adkv_oracle as orc
from tests.test_gpu_segments import _logit_errors
from tests.test_gpu_tail_state import ATOL, RTOL, _bits_equal, _oracle_tail, _prefill, _status_ok
from tests.util import SMAX, SMIN, dev, make_case, np_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("Hq,bits", [(2, 4), (4, 2), (8, 4), (8, 2)])
@pytest.mark.parametrize("T", [32, 33, 63, 64, 65, 79, 80, 81, 127, 128, 129, 193, 260])
def test_tile_edges(T, Hq, bits, pinned):
    case = make_case(1300 + T, 2, Hq, 2, T, bits)
    if pinned:
        for n in ("kp", "vp"):
            case[n][4][:, 5] = 100.0          # its scale falls to scale_min and stays there
    dk, dv, tk, tv, ok_, ov_, sk, sv = _prefill(case, T + 1)
    kn, vn = case["k"][:, :, T], case["v"][:, :, T]
    mask = torch.zeros(2, 1, 1, T + 1)
    mask[1, 0, 0, :T // 2] = torch.finfo(torch.float16).min
    for m in (mask, None):
        ok2, ov2 = ok_.copy(), ov_.copy()
        want = orc.decode_attn(case["q"][:, :, 0].numpy(), ok2, ov2, kn.numpy(), vn.numpy(), np_params(case["kp"]), np_params(case["vp"]),
                               T, 0.08, mask=None if m is None else m[:, 0].numpy(), bits=bits, scale_min=SMIN, scale_max=SMAX)
        got = gemv.decode_attn(dev(case["q"]), dk, dv, dev(kn[:, :, None]), dev(vn[:, :, None]), dev(case["kp"]), dev(case["vp"]), T,
                               0.08, SMIN, SMAX, mask=None if m is None else dev(m), bits=bits, k_tail=tk, v_tail=tv, tail_keep=m is not None)
        _status_ok()
        np.testing.assert_allclose(got.float().cpu().numpy(), want, rtol=RTOL, atol=ATOL)
        assert np.array_equal(dk.cpu().numpy(), ok2) and np.array_equal(dv.cpu().numpy(), ov2)
    orc.append_token(ok_, kn.numpy(), sk, T, np_params(case["kp"]), bits, SMIN, SMAX)
    orc.append_token(ov_, vn.numpy(), sv, T, np_params(case["vp"]), bits, SMIN, SMAX)
    assert _bits_equal(tk, _oracle_tail(sk)) and _bits_equal(tv, _oracle_tail(sv))


def _filled(case, B, H, T, smin, smax, bits, ckpt=0):
    kp, vp = dev(case["kp"]), dev(case["vp"])
    kc = torch.zeros(orc.cache_shape(B, H, orc.n_super_for(T + 1, bits), 128), dtype=torch.uint8, device="cuda")
    vc = torch.zeros_like(kc)
    kt, vt = torch.zeros(B, H, 2, 128, device="cuda"), torch.zeros(B, H, 2, 128, device="cuda")
    extra = {}
    if ckpt:
        kk, vk = (gemv.alloc_ckpt(B, H, 128, T + 1, ckpt, "cuda") for _ in range(2))
        extra = dict(k_ckpt=kk, v_ckpt=vk, ckpt_interval=ckpt)
    gemv.encode_kv_pair(kc, dev(case["k"][:, :, :T]), kp, vc, dev(case["v"][:, :, :T]), vp, smin, smax, bits=bits, k_tail=kt, v_tail=vt,
                        **extra)
    args = (dev(case["q"]), kc, vc, dev(case["k"][:, :, T:]), dev(case["v"][:, :, T:]), kp, vp)
    return args, dict(bits=bits, k_tail=kt, v_tail=vt, tail_keep=True), extra


@pytest.mark.parametrize("T,interval,Hq,bits", [(127, 64, 4, 4), (128, 64, 8, 2), (191, 96, 2, 4), (300, 96, 8, 4), (255, 128, 2, 2), (95, 32, 4, 2)])
def test_checkpoint_segments(T, interval, Hq, bits):
    """Segments that end inside a tile, an empty last segment, and the checkpoint that the appended token completes."""
    case = make_case(1500 + T, 2, Hq, 2, T, bits)
    args, kw, ck = _filled(case, 2, 2, T, SMIN, SMAX, bits, interval)
    want = gemv.decode_attn(*args, T, 0.08, SMIN, SMAX, **kw, split_channels=False)
    kw["tail_keep"] = False
    got = gemv.decode_attn(*args, T, 0.08, SMIN, SMAX, **kw, **ck)
    _status_ok()
    np.testing.assert_allclose(got.float().cpu().numpy(), want.float().cpu().numpy(), rtol=RTOL, atol=ATOL)
    if (T + 1) % interval == 0:
        n = (T + 1) // interval - 1
        assert _bits_equal(ck["k_ckpt"][:, :, n], kw["k_tail"].cpu().numpy()) and _bits_equal(ck["v_ckpt"][:, :, n], kw["v_tail"].cpu().numpy())


@pytest.mark.parametrize("kind", ["large", "small", "tiny_bounds", "zero_start", "large_first_value", "fast_zero_point", "zero_query", "large_query"])
@pytest.mark.parametrize("Hq,bits", [(2, 2), (8, 4)])
def test_ranges(Hq, bits, kind):
    """Scales of thousands, of 1e-5, of the quantiser's eps, from zero, one beyond scale_max in the first token; alpha above one; queries at either end: as the scan with fp32 sums gives it, in units of
    the result."""
    T, smin, smax, scaling = 150, SMIN, SMAX, 0.08
    case = make_case(1700, 2, Hq, 2, T, bits)
    k, v, q = case["k"], case["v"], case["q"]
    for n in ("kp", "vp"):
        zp, sc, al, be, tg = (t.clone() for t in case[n])
        if kind == "large":
            smin, smax = 4.0, 30000.0
            sc[:, ::3] = 9000.0
        elif kind == "small":
            smin, smax = 1e-6, 2.0 ** -7
            sc[:] = 2e-5
        elif kind == "tiny_bounds":
            smin, smax = 1e-10, 1e-9          # below the quantiser's eps, by which the values go then
            zp[:], sc[:] = 1.0, 0.0
        elif kind == "large_first_value":
            sc[:, ::7] = 50000.0
        elif kind == "zero_start":
            sc[:, ::4] = 0.0
        elif kind == "fast_zero_point":
            al[:, ::5] = 1.5
        case[n] = (zp, sc, al, be, tg)
    if kind == "large":
        case["k"], case["v"], scaling = (k.float().clamp(-100, 100) * 600).half(), (v.float().clamp(-100, 100) * 600).half(), 1e-5
    elif kind == "small":
        case["k"], case["v"], scaling = (k.float() * 2e-5).half(), (v.float() * 2e-5).half(), 2000.0
    elif kind == "large_first_value":         # the code of the large scale is one
        k[:, :, 0, ::7], v[:, :, 0, ::7], scaling = 60000.0, 60000.0, 1e-5
    elif kind == "zero_query":
        case["q"] = torch.zeros_like(q)
    elif kind == "large_query":
        case["q"], scaling = (q.float() * 10000).clamp(-60000, 60000).half(), 8e-6
    args, kw, _ = _filled(case, 2, 2, T, smin, smax, bits)
    want = gemv.decode_attn(*args, T, scaling, smin, smax, **kw, split_channels=False).float().cpu().numpy()
    got = gemv.decode_attn(*args, T, scaling, smin, smax, **kw).float().cpu().numpy()
    _status_ok()
    assert np.isfinite(want).all()
    np.testing.assert_allclose(got, want, rtol=RTOL, atol=ATOL * np.abs(want).max())


@pytest.mark.parametrize("rising", [False, True])
@pytest.mark.parametrize("Hq,bits", [(32, 2), (32, 4), (128, 4)])
def test_bound_met_at_every_token(Hq, bits, rising):
    """One channel of every head meets a bound, a token later from head to head: each place of the 16 tokens between two votes."""
    H, T, smin, smax = 32, 100, 0.05, 2.0
    case = make_case(1950, 1, Hq, H, T, bits)
    for n, c in (("kp", 5), ("vp", 70)):
        zp, sc, al, be, tg = (t.clone() for t in case[n])
        be[:, c], tg[:, c] = 2 ** -6, -8.0 if rising else 8.0      # 12 % a token and up, 12 % and less down
        away = 1.125 ** (10 + torch.arange(H, dtype=torch.float32))
        sc[:, c] = (smax / away if rising else smin * away).to(sc.dtype)
        case[n] = (zp, sc, al, be, tg)
    args, kw, ck = _filled(case, 1, H, T, smin, smax, bits, 64)
    want = gemv.decode_attn(*args, T, 0.08, smin, smax, **kw, split_channels=False)
    outs = [gemv.decode_attn(*args, T, 0.08, smin, smax, **kw), gemv.decode_attn(*args, T, 0.08, smin, smax, **kw, **ck)]
    _status_ok()
    for got in outs:
        np.testing.assert_allclose(got.float().cpu().numpy(), want.float().cpu().numpy(), rtol=RTOL, atol=ATOL)


@pytest.mark.parametrize("T", [699, 700, 701])
def test_line_to_token_segments(T):
    """2-bit, one query head: the longest streams of this kernel and the shortest that are cut into segments; between checkpoints never."""
    case = make_case(1960, 1, 2, 2, T, 2)
    args, kw, ck = _filled(case, 1, 2, T, SMIN, SMAX, 2, 1024)
    want = gemv.decode_attn(*args, T, 0.08, SMIN, SMAX, **kw, split_channels=False)
    outs = [gemv.decode_attn(*args, T, 0.08, SMIN, SMAX, **kw), gemv.decode_attn(*args, T, 0.08, SMIN, SMAX, **kw, **ck)]
    _status_ok()
    for got in outs:
        np.testing.assert_allclose(got.float().cpu().numpy(), want.float().cpu().numpy(), rtol=RTOL, atol=ATOL)


@pytest.mark.parametrize("B,Hkv,Hq,T,bits", [(37, 8, 8, 260, 2), (40, 8, 32, 130, 4), (56, 8, 16, 300, 4), (93, 8, 32, 300, 2)])
def test_more_streams_than_a_round(B, Hkv, Hq, T, bits):
    """296, 320, 448 and 744 streams: two share an SM and its tensor memory, the others follow.  With device-side lengths these take
    one warp per tensor."""
    case = make_case(1800 + T, 1, Hq, Hkv, T, bits)
    (q, kc, vc, kn, vn, kp, vp), kw, _ = _filled(case, 1, Hkv, T, SMIN, SMAX, bits)
    rep = lambda t: t.repeat(B, *([1] * (t.dim() - 1)))
    want = gemv.decode_attn(q, kc, vc, kn, vn, kp, vp, T, 0.08, SMIN, SMAX, **kw, split_channels=False)
    many = (rep(q), rep(kc), rep(vc), rep(kn), rep(vn), kp, vp)
    kw.update(k_tail=rep(kw["k_tail"]), v_tail=rep(kw["v_tail"]))
    got = gemv.decode_attn(*many, T, 0.08, SMIN, SMAX, **kw)
    again = gemv.decode_attn_varlen(*many, torch.full((B,), T, dtype=torch.int32, device="cuda"), 0.08, SMIN, SMAX, **kw)
    _status_ok()
    for out in (got, again):
        np.testing.assert_allclose(out[:1].float().cpu().numpy(), want.float().cpu().numpy(), rtol=RTOL, atol=ATOL)
        assert torch.equal(out, rep(out[:1]))


# device-side lengths: up to a round of CTAs, more than that, sequences that are ranked by length (up to 128) and that are not
RAGGED = [(37, 4, 4, 2, 300), (60, 5, 2, 4, 600), (128, 4, 2, 2, 520), (129, 4, 4, 4, 560), (100, 7, 4, 2, 1100)]


@pytest.mark.parametrize("B,Hkv,G,bits,room", RAGGED)
def test_ragged_lengths(B, Hkv, G, bits, room):
    """Empty sequences, equal lengths, full caches, and one sequence past the capacity, which is reported and left alone; the others
    as the dense call on them alone gives it."""
    D, g = 128, torch.Generator().manual_seed(B)
    cap = gemv.n_super_for(room, bits) * (32 // bits)
    lens = torch.randint(0, room, (B,), generator=g)
    lens[::7] = lens[0]
    lens[1], lens[B - 2], lens[B // 2] = 0, cap - 1, cap
    kp, vp = (tuple(dev(p)) for p in (make_case(1, 1, Hkv, Hkv, 1, bits)[n] for n in ("kp", "vp")))
    shape = (B, Hkv, gemv.n_super_for(room, bits), D // 4, 4, 4)
    kc, vc = (torch.zeros(shape, dtype=torch.uint8, device="cuda") for _ in range(2))
    k, v = (torch.randn(B, Hkv, cap - 1, D, generator=torch.Generator("cuda").manual_seed(i), device="cuda").half() for i in (B, B + 1))
    gemv.encode_kv_pair(kc, k, kp, vc, v, vp, SMIN, SMAX, bits=bits)
    kt, vt = (torch.rand(B, Hkv, 2, D, generator=g).cuda() + 0.1 for _ in range(2))
    q = torch.randn(B, Hkv * G, 1, D, generator=g).half().cuda()
    kn, vn = (torch.randn(B, Hkv, 1, D, generator=g).half().cuda() for _ in range(2))
    refs = [x.clone() for x in (kc, vc, kt, vt)]
    got = gemv.decode_attn_varlen(q, kc, vc, kn, vn, kp, vp, lens.int().cuda(), 0.05, SMIN, SMAX, bits=bits, k_tail=kt, v_tail=vt)
    assert gemv.device_status() == 6 and gemv.device_status() == 0
    rest = [b for b in range(B) if b != B // 2]
    want = torch.empty_like(got)
    for b in rest:
        one = slice(b, b + 1)
        want[one] = gemv.decode_attn(q[one], refs[0][one], refs[1][one], kn[one], vn[one], kp, vp, int(lens[b]), 0.05, SMIN, SMAX, bits=bits,
                                     k_tail=refs[2][one], v_tail=refs[3][one], split_channels=False)
    _status_ok()
    np.testing.assert_allclose(got[rest].float().cpu().numpy(), want[rest].float().cpu().numpy(), rtol=RTOL, atol=ATOL)
    for a, b in zip((kc, vc, kt, vt), refs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("smax", [1e6, float("inf")])
@pytest.mark.parametrize("Hq,T,bits", [(2, 130, 4), (8, 300, 2), (4, 700, 4)])
def test_no_upper_bound(Hq, T, bits, smax):
    """Scales that may grow past what pairs of fp16 numbers hold: token segments, with fp32 values."""
    case = make_case(1900 + T, 1, Hq, 2, T, bits)
    args, kw, _ = _filled(case, 1, 2, T, SMIN, smax, bits)
    want = gemv.decode_attn(*args, T, 0.08, SMIN, smax, **kw, split_channels=False)
    got = gemv.decode_attn(*args, T, 0.08, SMIN, smax, **kw)
    _status_ok()
    np.testing.assert_allclose(got.float().cpu().numpy(), want.float().cpu().numpy(), rtol=RTOL, atol=ATOL)


# scale_init far above the scales that follow; bounds too far apart for one unit of fp16 pairs (then the scans with fp32 values);
# bounds as far apart as pairs may go, with scales at the lower one
FAR_SCALES = {"large_init": dict(init=60000.0), "wide_bounds": dict(smin=1e-6, smax=32768.0, gain=1000.0),
              "at_lower_bound": dict(smin=2.0 ** -7, smax=64.0, gain=50.0)}


@pytest.mark.parametrize("bits,G", [(4, 1), (4, 2), (4, 4), (2, 1), (2, 2), (2, 4)])
@pytest.mark.parametrize("scales", ["usual", *FAR_SCALES])
def test_logit_error_is_that_of_a_whole_scan(scales, bits, G):
    """No further from 64 bits than the scan with fp32 values."""
    pairs = [_logit_errors(64, 600, bits, False, (None, False), seed=s, G=G, **FAR_SCALES.get(scales, {})) for s in (5, 25, 45)]
    got, whole = (sum(e * e for e in errors) ** 0.5 for errors in zip(*pairs))
    # 576 logits; eight sets of 2000 tokens: 0.85 to 0.98, and 1.02 with every scale at the lower bound (4-bit), where no rounding
    # of a scale is carried on
    assert got <= whole * (1.05 if scales == "at_lower_bound" else 1.0), (got, whole)


@pytest.mark.parametrize("Hq,bits", [(2, 4), (8, 2)])
def test_step_that_gives_up_marks_its_result(Hq, bits):
    """With the K scan muted no sums of K ever come: every wait behind them runs out, the kernel ends by itself, nothing is appended
    and the output is NaN; the next call is as before."""
    T, interval, H = 496, 256, 2              # the appended token begins a word
    case = make_case(1980, 1, Hq, H, T, bits)
    args, kw, ck = _filled(case, 1, H, T, SMIN, SMAX, bits, interval)
    scratch = torch.empty(gemv.decode_scratch_bytes(1, Hq, H, T, interval), dtype=torch.uint8, device="cuda")
    good = gemv.decode_attn(*args, T, 0.08, SMIN, SMAX, **kw, **ck, scratch=scratch)
    _status_ok()
    q, kc, vc, kn, vn, kp, vp = args
    kt, vt, kk, vk = kw["k_tail"], kw["v_tail"], ck["k_ckpt"], ck["v_ckpt"]
    row = T // (32 // bits)
    kc[:, :, row], vc[:, :, row] = 0, 0
    before = [t.clone() for t in (kc, vc, kt, vt, kk, vk)]
    out = torch.zeros_like(good)
    pk, pv = (_lib.Params(*[t.data_ptr() for t in ps]) for ps in (kp, vp))
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    rc = _lib.load().adkv_decode_attn_ckpt(
        q.data_ptr(), kc.data_ptr(), vc.data_ptr(), kn.data_ptr(), vn.data_ptr(), ctypes.addressof(pk), ctypes.addressof(pv),
        kt.data_ptr(), vt.data_ptr(), kk.data_ptr(), vk.data_ptr(), interval, kk.shape[2], None, 0, out.data_ptr(), scratch.data_ptr(),
        scratch.numel(), 1, Hq, H, T, 128, kc.shape[2], bits, 0.08, SMIN, SMAX, _lib.FLAG_SELFTEST_MUTE_K | _lib.FLAG_FAST_REPLAY,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    seconds = time.perf_counter() - t0
    assert 1 <= gemv.device_status() <= 4
    assert torch.isnan(out).all()
    for t, old in zip((kc, vc, kt, vt, kk, vk), before):
        assert torch.equal(t, old)
    assert 0.9 < seconds < 4.0, seconds      # 2e9 cycles at 1.965 GHz or less
    again = gemv.decode_attn(*args, T, 0.08, SMIN, SMAX, **kw, **ck, scratch=scratch)
    _status_ok()
    assert torch.equal(again, good)
