"""Decode steps next to tail states against the oracle and against 64 bits: what the library picks for few streams (the tensor
cores, but for 2-bit codes of one query head from 700 tokens on), token segments (the same streams of 128 tokens and more,
any device-side length, where the scale bounds are too far apart for the tensor cores), and one warp pair per stream; prefill and
append by number of streams.  Needs a B200.

Sizes are the edges of the split: no token, fewer tiles than segments, whole tiles, one token more or less; scales that
never clamp, clamp at one bound, at both, and start outside the bounds.  test_launches.py holds which kernel a call takes.
"""
import numpy as np
import pytest
import torch

from adkv_b200 import gemv, synth
from oracle import adkv_oracle as orc
from tests.test_gpu_tail_state import ATOL, RTOL, _bits_equal, _oracle_tail, _prefill, _status_ok
from tests.util import SMAX, SMIN, WIDE, dev, make_case, np_params

pytestmark = pytest.mark.gpu


def _clamping(case, kind):
    """Parameters under which the scales meet the clamp bounds."""
    for n in ("kp", "vp"):
        zp, sc, al, be, tg = (t.clone() for t in case[n])
        if kind == "pinned_low":
            tg[:, ::3] = 7.5        # mean code magnitude never reached: these scales fall to scale_min and stay there
        elif kind == "both":
            be[:, ::2] = 0.45       # growth factors far from 1: both bounds within a few tokens
        elif kind == "start_outside":
            sc[:, ::5] = 0.0
            sc[:, 1::5] = 100.0
        elif kind == "odd_factor":
            be[:, ::7] = 0.9
            tg[:, ::7] = 4.0        # 1 - beta * target < 0
        case[n] = (zp, sc, al, be, tg)


BOUNDS = {"usual": (SMIN, SMAX), "wide": WIDE}
SHAPES = [
    (1, 2, 2, 0, 4), (1, 2, 2, 1, 2), (2, 2, 2, 31, 4), (1, 4, 2, 32, 4), (1, 4, 1, 33, 2), (2, 2, 2, 255, 4), (1, 2, 1, 256, 2),
    (1, 2, 2, 257, 4), (1, 8, 2, 290, 2), (1, 2, 2, 777, 2), (2, 4, 2, 1031, 4),
    (1, 2, 2, 127, 4), (1, 4, 2, 128, 2), (1, 2, 2, 129, 4), (1, 8, 2, 225, 4),
]


@pytest.mark.parametrize("bounds,split", [("usual", None), ("wide", None), ("usual", False)], ids=["library", "segments", "whole_head"])
@pytest.mark.parametrize("clamp", ["none", "pinned_low", "both", "start_outside", "odd_factor"])
@pytest.mark.parametrize("B,Hq,Hkv,T,bits", SHAPES)
def test_against_oracle(B, Hq, Hkv, T, bits, clamp, bounds, split):
    smin, smax = BOUNDS[bounds]
    case = make_case(500 + T, B, Hq, Hkv, T, bits)
    _clamping(case, clamp)
    dk, dv, tk, tv, ok_, ov_, sk, sv = _prefill(case, T + 1, (smin, smax))
    kn, vn = case["k"][:, :, T], case["v"][:, :, T]
    mask = torch.zeros(B, 1, 1, T + 1)
    mask[0, 0, 0, :T // 3] = torch.finfo(torch.float16).min
    variants = {"mask": mask, "plain": None}
    for name, m in variants.items():
        ok2, ov2 = ok_.copy(), ov_.copy()
        want = orc.decode_attn(case["q"][:, :, 0].numpy(), ok2, ov2, kn.numpy(), vn.numpy(), np_params(case["kp"]),
                               np_params(case["vp"]), T, 0.07, mask=None if m is None else m[:, 0].numpy(), bits=bits,
                               scale_min=smin, scale_max=smax)
        got = gemv.decode_attn(dev(case["q"]), dk, dv, dev(kn[:, :, None]), dev(vn[:, :, None]), dev(case["kp"]), dev(case["vp"]),
                               T, 0.07, smin, smax, mask=None if m is None else dev(m), bits=bits, k_tail=tk, v_tail=tv,
                               tail_keep=name == "mask", split_channels=split)
        _status_ok()
        np.testing.assert_allclose(got.float().cpu().numpy(), want, rtol=RTOL, atol=ATOL)
        assert np.array_equal(dk.cpu().numpy(), ok2) and np.array_equal(dv.cpu().numpy(), ov2)
    orc.append_token(ok_.copy(), kn.numpy(), sk, T, np_params(case["kp"]), bits, smin, smax)
    orc.append_token(ov_.copy(), vn.numpy(), sv, T, np_params(case["vp"]), bits, smin, smax)
    assert _bits_equal(tk, _oracle_tail(sk)) and _bits_equal(tv, _oracle_tail(sv))


@pytest.mark.parametrize("bounds", BOUNDS)
@pytest.mark.parametrize("bits", [4, 2])
def test_segments_varlen(bits, bounds):
    """Ragged lengths, one of them zero: every sequence as the dense call on it alone gives it."""
    smin, smax = BOUNDS[bounds]
    B, Hq, Hkv, D, lens = 3, 4, 2, 128, [0, 97, 640]
    case = make_case(77, B, Hq, Hkv, max(lens), bits)
    ns = orc.n_super_for(max(lens) + 1, bits)
    dk = torch.zeros(orc.cache_shape(B, Hkv, ns, D), dtype=torch.uint8, device="cuda")
    dv = torch.zeros_like(dk)
    tk = torch.zeros(B, Hkv, 2, D, device="cuda")
    tv = torch.zeros_like(tk)
    kp, vp = dev(case["kp"]), dev(case["vp"])
    for b, n in enumerate(lens):
        gemv.encode_kv_pair(dk[b:b + 1], dev(case["k"][b:b + 1, :, :n]), kp, dv[b:b + 1], dev(case["v"][b:b + 1, :, :n]), vp,
                            smin, smax, bits=bits, k_tail=tk[b:b + 1], v_tail=tv[b:b + 1])
    kn, vn = dev(case["k"][:, :, -1:]), dev(case["v"][:, :, -1:])
    q = dev(case["q"])
    want = torch.cat([gemv.decode_attn(q[b:b + 1], dk[b:b + 1].clone(), dv[b:b + 1].clone(), kn[b:b + 1], vn[b:b + 1], kp, vp, n,
                                       0.09, smin, smax, bits=bits, k_tail=tk[b:b + 1], v_tail=tv[b:b + 1], tail_keep=True,
                                       split_channels=False) for b, n in enumerate(lens)])
    got = gemv.decode_attn_varlen(q, dk, dv, kn, vn, kp, vp, torch.tensor(lens, dtype=torch.int32, device="cuda"), 0.09, smin,
                                  smax, bits=bits, k_tail=tk, v_tail=tv)
    _status_ok()
    np.testing.assert_allclose(got.float().cpu().numpy(), want.float().cpu().numpy(), rtol=RTOL, atol=ATOL)


@pytest.mark.parametrize("bounds", BOUNDS)
@pytest.mark.parametrize("Hq,Hkv,bits", [(2, 2, 4), (8, 2, 2)])
def test_segments_varlen_short(Hq, Hkv, bits, bounds):
    """Sequences from one token to a few tiles, and one past the capacity, in caches with room for 700: one tile is
    one segment.  The sequence that does not fit is reported and left alone."""
    smin, smax = BOUNDS[bounds]
    lens, D = [1, 32, 33, 95, 96, 97, 128, 129, 224, 225, 700], 128
    B, cap = len(lens), 700
    case = make_case(78, B, Hq, Hkv, cap, bits)
    dk = torch.zeros(orc.cache_shape(B, Hkv, orc.n_super_for(cap, bits), D), dtype=torch.uint8, device="cuda")
    dv = torch.zeros_like(dk)
    tk = torch.zeros(B, Hkv, 2, D, device="cuda")
    tv = torch.zeros_like(tk)
    kp, vp = dev(case["kp"]), dev(case["vp"])
    for b, n in enumerate(lens):
        gemv.encode_kv_pair(dk[b:b + 1], dev(case["k"][b:b + 1, :, :n]), kp, dv[b:b + 1], dev(case["v"][b:b + 1, :, :n]), vp,
                            smin, smax, bits=bits, k_tail=tk[b:b + 1], v_tail=tv[b:b + 1])
    lens[-1] = dk.shape[2] * (32 // bits)
    kn, vn, q = dev(case["k"][:, :, -1:]), dev(case["v"][:, :, -1:]), dev(case["q"])
    before = [t.clone() for t in (dk, dv, tk, tv)]
    want = torch.cat([gemv.decode_attn(q[b:b + 1], dk[b:b + 1].clone(), dv[b:b + 1].clone(), kn[b:b + 1], vn[b:b + 1], kp, vp, n,
                                       0.09, smin, smax, bits=bits, k_tail=tk[b:b + 1], v_tail=tv[b:b + 1], tail_keep=True,
                                       split_channels=False) for b, n in enumerate(lens[:-1])])
    got = gemv.decode_attn_varlen(q, dk, dv, kn, vn, kp, vp, torch.tensor(lens, dtype=torch.int32, device="cuda"), 0.09, smin,
                                  smax, bits=bits, k_tail=tk, v_tail=tv)
    assert gemv.device_status() == 6 and gemv.device_status() == 0
    np.testing.assert_allclose(got[:-1].float().cpu().numpy(), want.float().cpu().numpy(), rtol=RTOL, atol=ATOL)
    for t, old in zip((dk, dv, tk, tv), before):
        assert torch.equal(t[-1], old[-1])


@pytest.mark.parametrize("bounds", BOUNDS)
@pytest.mark.parametrize("Hq,T,bits", [(2, 300, 4), (8, 531, 2)])
def test_masked_segments(Hq, T, bits, bounds):
    """Additive masks that leave out whole segments, every cached token, and everything; the lowest fp32 and fp16 values
    as well as minus infinity."""
    smin, smax = BOUNDS[bounds]
    case = make_case(610, 1, Hq, 2, T, bits)
    dk, dv, tk, tv, *_ = _prefill(case, T + 1, (smin, smax))
    args = (dev(case["q"]), dk, dv, dev(case["k"][:, :, T:]), dev(case["v"][:, :, T:]), dev(case["kp"]), dev(case["vp"]), T, 0.08,
            smin, smax)
    kw = dict(bits=bits, k_tail=tk, v_tail=tv, tail_keep=True)
    for low in (-float("inf"), torch.finfo(torch.float32).min, torch.finfo(torch.float16).min):
        for out in (slice(0, T // 2), slice(T // 4, T), slice(0, T), slice(0, T + 1)):
            mask = torch.zeros(1, T + 1, device="cuda")
            mask[:, out] = low
            want = gemv.decode_attn(*args, **kw, mask=mask, split_channels=False)
            got = gemv.decode_attn(*args, **kw, mask=mask)
            if out == slice(0, T + 1) and low > -1e5:    # scores near -94500 are an fp32 unit of 2**-7 apart, and are
                rtol = atol = 2e-2                       # rounded twice: weights to 2 * 2**-7 * ln 2
            else:
                rtol, atol = RTOL, ATOL
            np.testing.assert_allclose(got.float().cpu().numpy(), want.float().cpu().numpy(), rtol=rtol, atol=atol)
    _status_ok()


def test_product_past_the_range_of_fp32():
    """Factors far above 1 and no lower bound: the product of a segment's factors overflows, its scales end at the upper
    bound."""
    T, bits, smax = 700, 4, 4.0
    case = make_case(620, 1, 2, 2, T, bits)
    for n in ("kp", "vp"):
        be, tg = case[n][3].clone(), case[n][4].clone()
        be[:, ::3], tg[:, ::3] = 8.0, 0.0
        case[n] = (*case[n][:3], be, tg)
    dk = torch.zeros(orc.cache_shape(1, 2, orc.n_super_for(T + 1, bits), 128), dtype=torch.uint8, device="cuda")
    dv = torch.zeros_like(dk)
    tk, tv = torch.zeros(1, 2, 2, 128, device="cuda"), torch.zeros(1, 2, 2, 128, device="cuda")
    kp, vp = dev(case["kp"]), dev(case["vp"])
    gemv.encode_kv_pair(dk, dev(case["k"][:, :, :T]), kp, dv, dev(case["v"][:, :, :T]), vp, 0.0, smax, bits=bits, k_tail=tk, v_tail=tv)
    args = (dev(case["q"]), dk, dv, dev(case["k"][:, :, T:]), dev(case["v"][:, :, T:]), kp, vp, T, 0.05, 0.0, smax)
    kw = dict(bits=bits, k_tail=tk, v_tail=tv, tail_keep=True)
    want, got = gemv.decode_attn(*args, **kw, split_channels=False), gemv.decode_attn(*args, **kw)
    _status_ok()
    assert torch.isfinite(want.float()).all()
    np.testing.assert_allclose(got.float().cpu().numpy(), want.float().cpu().numpy(), rtol=RTOL, atol=ATOL)


def test_layered_append_forms():
    """33 layers (one more than a launch takes): stacked buffers, lists of tensors and pointers that are only aligned to
    their type give the bytes and states of one append per layer."""
    L, B, H, D, T, bits = 33, 1, 3, 128, 37, 4
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    shape = (L, B, H, orc.n_super_for(T + 1, bits), D // 4, 4, 4)
    base = torch.randint(0, 256, shape, generator=g, device="cuda", dtype=torch.uint8)
    tails = rnd(2, L, B, H, 2, D)
    tails[:, :, :, :, 1] = tails[:, :, :, :, 1].abs() + 0.1
    params = [[tuple(t.half().abs() * 0.3 for t in rnd(5, H, D)) for _ in range(2)] for _ in range(L)]
    x = rnd(2, L, B, H, D).half()

    def fresh():
        return base.clone(), base.clone(), tails[0].clone(), tails[1].clone()

    kc, vc, kt, vt = want = fresh()
    for i in range(L):
        gemv.append_kv_pair(kc[i], x[0, i][:, :, None], params[i][0], kt[i], vc[i], x[1, i][:, :, None], params[i][1], vt[i], T,
                            SMIN, SMAX, bits=bits)
    odd = torch.empty(x.numel() + 1, dtype=torch.float16, device="cuda")[1:].view_as(x)   # 2 bytes off
    odd.copy_(x)
    for k, v in ((x[0], x[1]), (list(x[0].unbind()), list(x[1].unbind())), (odd[0], odd[1])):
        kc, vc, kt, vt = got = fresh()
        ls = gemv.LayerSet([(kc[i], params[i][0], kt[i], vc[i], params[i][1], vt[i]) for i in range(L)], bits=bits)
        gemv.append_kv_layers(ls, k, v, T, SMIN, SMAX)
        for a, b in zip(got, want):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    with pytest.raises(RuntimeError, match="wrong shape"):
        gemv.append_kv_layers(ls, x[0, :, :, :2].contiguous(), x[1], T, SMIN, SMAX)


@pytest.mark.parametrize("Hq,Hkv,T,bits", [(2, 2, 0, 4), (2, 2, 95, 4), (8, 2, 129, 2), (4, 2, 300, 4)])
def test_two_streams_per_sm(Hq, Hkv, T, bits):
    """160 streams, more than the segments take: what the library picks and split heads, against one warp pair per stream."""
    B, D = 80, 128
    case = make_case(900 + T, 2, Hq, Hkv, T, bits)
    dk, dv, tk, tv, ok_, ov_, *_ = _prefill(case, T + 1)
    rep = lambda t: dev(t).repeat(B // 2, *([1] * (t.dim() - 1)))
    args = (rep(case["q"]), rep(dk), rep(dv), rep(case["k"][:, :, T:]), rep(case["v"][:, :, T:]), dev(case["kp"]), dev(case["vp"]),
            T, 0.08, SMIN, SMAX)
    kw = dict(bits=bits, k_tail=rep(tk), v_tail=rep(tv), tail_keep=True)
    want = gemv.decode_attn(*args, **kw, split_channels=False)
    for split in (None, True):
        got = gemv.decode_attn(*args, **kw, split_channels=split)
        _status_ok()
        np.testing.assert_allclose(got.float().cpu().numpy(), want.float().cpu().numpy(), rtol=RTOL, atol=ATOL)
        assert torch.equal(got[:2], got[-2:])


@pytest.mark.parametrize("T,bits", [(1, 4), (33, 4), (70, 2)])
def test_few_and_many_streams_agree(T, bits):
    """Prefill (one or two channels per thread) and forward_ov (one or two warps per stream) choose by the number of streams;
    bytes, states and outputs do not depend on it."""
    B, H, D = 160, 4, 128
    case = make_case(40 + T, 1, H, H, T, bits)
    dk, dv, tk, tv, *_ = _prefill(case, T + 1)
    rep = lambda t: dev(t).repeat(B, *([1] * (t.dim() - 1)))
    mk, mv, mtk, mtv = torch.zeros_like(rep(dk)), torch.zeros_like(rep(dv)), torch.zeros_like(rep(tk)), torch.zeros_like(rep(tv))
    kp, vp = dev(case["kp"]), dev(case["vp"])
    gemv.encode_kv_pair(mk, rep(case["k"][:, :, :T]), kp, mv, rep(case["v"][:, :, :T]), vp, SMIN, SMAX, bits=bits, k_tail=mtk,
                        v_tail=mtv)
    for many, one in ((mk, dk), (mv, dv), (mtk, tk), (mtv, tv)):
        assert torch.equal(many.view(torch.uint8), rep(one).view(torch.uint8))
    w = torch.softmax(torch.randn(1, H, T + 1, generator=torch.Generator().manual_seed(1)), -1).half()
    one = gemv.forward_ov(dev(w), dv, dev(case["v"][:, :, T:]), *vp, SMIN, SMAX, bits=bits)
    many = gemv.forward_ov(rep(w), mv, rep(case["v"][:, :, T:]), *vp, SMIN, SMAX, bits=bits)
    assert torch.equal(many, rep(one)) and torch.equal(mv, rep(dv))
    _status_ok()


def _replay64(cache, params, T, at, bits, smin=SMIN, smax=SMAX):
    """The recurrence in 64 bits over the stored codes: values of the tokens in ``at``, [len(at), streams, 128]."""
    B, H = cache.shape[:2]
    words = cache.view(B * H, -1, 128 * 4).contiguous().view(torch.int32)
    tpw, bias = 32 // bits, 1 << (bits - 1)
    zp, s, al, be, tg = (p.double().repeat(B, 1) for p in params)
    out = []
    for t in range(T):
        q = ((words[:, t // tpw] >> (bits * (t % tpw))) & ((1 << bits) - 1)).double() - bias
        rh = q * s.clamp(min=1e-8)
        if t in at:
            out.append(zp + rh)
        zp = zp + al * rh
        s = (s * (1.0 - be * tg + be * q.abs())).clamp(smin, smax)
    return torch.stack(out)


def _logit_errors(B, T, bits, pinned, variants, seed=5, G=1, smin=SMIN, smax=SMAX, init=None, gain=1.0):
    """Root mean square error of single logits against 64 bits, one figure per entry of ``variants`` (split_channels).
    G query heads, all alike; ``init``: scale_init of every fourth channel; ``gain``: K and its scales are made smaller by
    it and q larger.

    A mask leaves one cached token and the appended one, and cancels the cached token's exact logit against the appended
    token's; the scaling magnifies what remains.  The output is then v_self + a * (v_cached - v_self), where a / (1 - a) is
    the exponential of the magnified error of that one logit.
    """
    D, scaling = 128, 2000.0
    k, v = (synth.gen_kv(seed + i, B, 1, T + 1, D, device="cuda") for i in (0, 1))
    q = (synth.gen_q(seed + 2, B, 1, D, device="cuda") * gain).expand(B, G, 1, D).contiguous()
    k = k / gain
    kp, vp = (synth.gen_params(seed + 3 + i, 1, D, bits, device="cuda") for i in (0, 1))
    kp[1].div_(gain)
    if init is not None:
        kp[1][:, ::4] = init
    if pinned:      # one channel of the head whose scale rests at scale_min
        kp[4][:, 17] = float(1 << (bits - 1))
        vp[4][:, 17] = float(1 << (bits - 1))
    kc = torch.zeros(orc.cache_shape(B, 1, orc.n_super_for(T + 1, bits), D), dtype=torch.uint8, device="cuda")
    vc = torch.zeros_like(kc)
    kt, vt = torch.zeros(B, 1, 2, D, device="cuda"), torch.zeros(B, 1, 2, D, device="cuda")
    gemv.encode_kv_pair(kc, k[:, :, :T], kp, vc, v[:, :, :T], vp, smin, smax, bits=bits, k_tail=kt, v_tail=vt)
    at = sorted({T - 1, T - T // 8 - 1, T // 2 + 5})
    kx, vx = _replay64(kc, kp, T, at, bits, smin, smax), _replay64(vc, vp, T, at, bits, smin, smax)

    def appended(cache, tail):     # the appended token, from the tail it is quantised with
        word = cache.view(B, -1, D * 4).contiguous().view(torch.int32)[:, T // (32 // bits)]
        code = ((word >> (bits * (T % (32 // bits)))) & ((1 << bits) - 1)).double() - (1 << (bits - 1))
        return tail[:, 0, 0].double() + code * tail[:, 0, 1].double().clamp(min=1e-8)

    errors = []
    for split in variants:
        sq, n = 0.0, 0
        for i, t in enumerate(at):
            args = (q, kc, vc, k[:, :, T:], v[:, :, T:], kp, vp, T, scaling, smin, smax)
            kw = dict(bits=bits, k_tail=kt, v_tail=vt, tail_keep=True, split_channels=split)
            gemv.decode_attn(*args, **kw)      # writes the appended codes
            ks, vs = appended(kc, kt), appended(vc, vt)
            qd = q[:, 0, 0].double()
            mask = torch.full((B, T + 1), -float("inf"), device="cuda")
            mask[:, T] = 0.0
            shift = (scaling * (qd * (ks - kx[i])).sum(-1)).float()
            mask[:, t] = shift
            out = gemv.decode_attn(*args, mask=mask, **kw).double()
            d = (vx[i] - vs)[:, None]
            a = ((out - vs[:, None]) * d).sum(-1) / (d * d).sum(-1)
            left = scaling * (qd * (kx[i] - ks)).sum(-1) + shift.double()     # what the rounding of the mask leaves
            err = (torch.log(a / (1.0 - a)) - left[:, None]) / scaling
            sq, n = sq + float((err * err).sum()), n + err.numel()
        errors.append((sq / n) ** 0.5)
    _status_ok()
    return errors


@pytest.mark.parametrize("bounds", BOUNDS)
@pytest.mark.parametrize("B,T,bits,pinned", [(64, 4096, 2, False), (128, 8192, 2, False), (64, 2000, 4, False), (128, 4096, 4, False),
                                             (64, 4096, 4, True), (64, 8192, 2, True)])
def test_logit_error_is_that_of_a_whole_scan(B, T, bits, pinned, bounds):
    """Segments start from products of their predecessors' factors, the tensor cores sum pairs of fp16 numbers: no further from
    64 bits than one scan over the stream.  Sums of 192 to 384 squared errors each; segments start from less rounding, which
    leaves 0.6 to 0.85 of the whole scan's."""
    smin, smax = BOUNDS[bounds]
    got, whole = _logit_errors(B, T, bits, pinned, (None, False), smin=smin, smax=smax)
    assert got <= whole, (got, whole)


@pytest.mark.parametrize("T,bits", [(70, 4), (161, 2)])
def test_checkpoints_of_few_and_many_streams(T, bits):
    """Checkpoints, codes and tails of a prefill with a channel pair per thread (more than 444 (stream, tensor) pairs) are
    those of the one-channel form, bit for bit; started inside a word as well as at the front."""
    B, H, D, S = 160, 2, 128, 32
    case = make_case(50 + T, 1, H, H, T, bits)
    kp, vp = dev(case["kp"]), dev(case["vp"])

    def prefill(n):
        rep = lambda t: dev(t).repeat(n, 1, 1, 1)
        kc = torch.zeros(orc.cache_shape(n, H, orc.n_super_for(T, bits), D), dtype=torch.uint8, device="cuda")
        vc, kt, vt = torch.zeros_like(kc), torch.zeros(n, H, 2, D, device="cuda"), torch.zeros(n, H, 2, D, device="cuda")
        kk, vk = gemv.alloc_ckpt(n, H, D, T, S, "cuda"), gemv.alloc_ckpt(n, H, D, T, S, "cuda")
        for lo, hi in ((0, 37), (37, T)):
            gemv.encode_kv_pair(kc, rep(case["k"][:, :, lo:hi]), kp, vc, rep(case["v"][:, :, lo:hi]), vp, SMIN, SMAX, bits=bits,
                                t_start=lo, k_tail=kt, v_tail=vt, k_ckpt=kk, v_ckpt=vk, ckpt_interval=S)
        return kc, vc, kt, vt, kk, vk

    for many, one in zip(prefill(B), prefill(1)):
        assert torch.equal(many.view(torch.uint8), one.repeat(B, *([1] * (one.dim() - 1))).view(torch.uint8))
    assert float(one[:, :, -1, 1].min()) > 0.0      # the last checkpoint is written
