"""Decode steps next to tail states against the oracle, over token segments (launches with few streams) and with one
warp pair per stream.  Needs a B200.

Sizes are the edges of the split: no token, fewer tiles than segments, whole tiles, one token more or less; scales that
never clamp, clamp at one bound, at both, and start outside the bounds.
"""
import numpy as np
import pytest
import torch

from adkv_b200 import gemv
from oracle import adkv_oracle as orc
from tests.test_gpu_tail_state import ATOL, RTOL, _bits_equal, _oracle_tail, _prefill, _status_ok
from tests.util import SMAX, SMIN, dev, make_case, np_params

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


@pytest.mark.parametrize("split", [None, False], ids=["segments", "whole_head"])
@pytest.mark.parametrize("clamp", ["none", "pinned_low", "both", "start_outside", "odd_factor"])
@pytest.mark.parametrize("B,Hq,Hkv,T,bits", [
    (1, 2, 2, 0, 4), (1, 2, 2, 1, 2), (2, 2, 2, 31, 4), (1, 4, 2, 32, 4), (1, 4, 1, 33, 2), (2, 2, 2, 255, 4), (1, 2, 1, 256, 2),
    (1, 2, 2, 257, 4), (1, 8, 2, 290, 2), (1, 2, 2, 777, 2), (2, 4, 2, 1031, 4),
])
def test_against_oracle(B, Hq, Hkv, T, bits, clamp, split):
    case = make_case(500 + T, B, Hq, Hkv, T, bits)
    _clamping(case, clamp)
    dk, dv, tk, tv, ok_, ov_, sk, sv = _prefill(case, T + 1)
    kn, vn = case["k"][:, :, T], case["v"][:, :, T]
    mask = torch.zeros(B, 1, 1, T + 1)
    mask[0, 0, 0, :T // 3] = torch.finfo(torch.float16).min
    variants = {"mask": mask, "plain": None}
    for name, m in variants.items():
        ok2, ov2 = ok_.copy(), ov_.copy()
        want = orc.decode_attn(case["q"][:, :, 0].numpy(), ok2, ov2, kn.numpy(), vn.numpy(), np_params(case["kp"]),
                               np_params(case["vp"]), T, 0.07, mask=None if m is None else m[:, 0].numpy(), bits=bits,
                               scale_min=SMIN, scale_max=SMAX)
        got = gemv.decode_attn(dev(case["q"]), dk, dv, dev(kn[:, :, None]), dev(vn[:, :, None]), dev(case["kp"]), dev(case["vp"]),
                               T, 0.07, SMIN, SMAX, mask=None if m is None else dev(m), bits=bits, k_tail=tk, v_tail=tv,
                               tail_keep=name == "mask", split_channels=split)
        _status_ok()
        np.testing.assert_allclose(got.float().cpu().numpy(), want, rtol=RTOL, atol=ATOL)
        assert np.array_equal(dk.cpu().numpy(), ok2) and np.array_equal(dv.cpu().numpy(), ov2)
    orc.append_token(ok_.copy(), kn.numpy(), sk, T, np_params(case["kp"]), bits, SMIN, SMAX)
    orc.append_token(ov_.copy(), vn.numpy(), sv, T, np_params(case["vp"]), bits, SMIN, SMAX)
    assert _bits_equal(tk, _oracle_tail(sk)) and _bits_equal(tv, _oracle_tail(sv))


@pytest.mark.parametrize("bits", [4, 2])
def test_segments_varlen(bits):
    """Ragged lengths, one of them zero: every sequence as the dense call on it alone gives it."""
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
                            SMIN, SMAX, bits=bits, k_tail=tk[b:b + 1], v_tail=tv[b:b + 1])
    kn, vn = dev(case["k"][:, :, -1:]), dev(case["v"][:, :, -1:])
    q = dev(case["q"])
    want = torch.cat([gemv.decode_attn(q[b:b + 1], dk[b:b + 1].clone(), dv[b:b + 1].clone(), kn[b:b + 1], vn[b:b + 1], kp, vp, n,
                                       0.09, SMIN, SMAX, bits=bits, k_tail=tk[b:b + 1], v_tail=tv[b:b + 1], tail_keep=True,
                                       split_channels=False) for b, n in enumerate(lens)])
    got = gemv.decode_attn_varlen(q, dk, dv, kn, vn, kp, vp, torch.tensor(lens, dtype=torch.int32, device="cuda"), 0.09, SMIN,
                                  SMAX, bits=bits, k_tail=tk, v_tail=tv)
    _status_ok()
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
    """160 streams: the eight-warp form of the segment kernel, against one warp pair per stream."""
    B, D = 80, 128
    case = make_case(900 + T, 2, Hq, Hkv, T, bits)
    dk, dv, tk, tv, ok_, ov_, *_ = _prefill(case, T + 1)
    rep = lambda t: dev(t).repeat(B // 2, *([1] * (t.dim() - 1)))
    args = (rep(case["q"]), rep(dk), rep(dv), rep(case["k"][:, :, T:]), rep(case["v"][:, :, T:]), dev(case["kp"]), dev(case["vp"]),
            T, 0.08, SMIN, SMAX)
    kw = dict(bits=bits, k_tail=rep(tk), v_tail=rep(tv), tail_keep=True)
    want = gemv.decode_attn(*args, **kw, split_channels=False)
    got = gemv.decode_attn(*args, **kw)
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
