"""Decode scans at the edges of their 64-token tiles, of the words in a ragged tile and of the checkpoint segments, against the
oracle.  Needs a B200."""
import numpy as np
import pytest
import torch

from adkv_b200 import gemv
from oracle import adkv_oracle as orc
from tests import test_gpu_half_state
from tests.test_gpu_tail_state import ATOL, RTOL, _prefill, _status_ok
from tests.util import SMAX, SMIN, WIDE, dev, make_case, np_params

pytestmark = pytest.mark.gpu

EDGES = [(1, 63), (1, 64), (2, 65), (1, 71), (4, 72), (1, 73), (2, 79), (4, 80), (1, 95), (1, 127), (4, 128), (1, 129)]


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("G,T", EDGES)
def test_against_oracle(G, T, bits):
    """One step as whole-head scans (contracted next to tails, canonical without), over checkpoints of 32 tokens, and as the
    three calls; all append the same codes."""
    B, Hkv = 2, 2
    case = make_case(900 + T, B, G * Hkv, Hkv, T, bits)
    case["kp"][4][:, ::5] = 7.5          # some scales rest at the lower bound
    ck = [gemv.alloc_ckpt(B, Hkv, 128, T + 1, 32, "cuda") for _ in range(2)]
    dk, dv, tk, tv, ok_, ov_, _, _ = _prefill(case, T + 1, k_ckpt=ck[0], v_ckpt=ck[1], ckpt_interval=32)
    kn, vn = case["k"][:, :, T], case["v"][:, :, T]
    mask = torch.zeros(B, T + 1)
    mask[0, :T // 3] = torch.finfo(torch.float16).min
    wk, wv = ok_.copy(), ov_.copy()
    want = orc.decode_attn(case["q"][:, :, 0].numpy(), wk, wv, kn.numpy(), vn.numpy(), np_params(case["kp"]),
                           np_params(case["vp"]), T, 0.07, mask=mask[:, None].numpy(), bits=bits, scale_min=SMIN, scale_max=SMAX)
    new = (dev(kn[:, :, None]), dev(vn[:, :, None]))
    kp, vp, q = dev(case["kp"]), dev(case["vp"]), dev(case["q"])
    for kw in (dict(k_tail=tk, v_tail=tv, tail_keep=True, split_channels=False), dict(split_channels=False),
               dict(k_tail=tk, v_tail=tv, tail_keep=True, k_ckpt=ck[0], v_ckpt=ck[1], ckpt_interval=32)):
        a, b = dk.clone(), dv.clone()
        got = gemv.decode_attn(q, a, b, *new, kp, vp, T, 0.07, SMIN, SMAX, mask=dev(mask), bits=bits, **kw)
        np.testing.assert_allclose(got.float().cpu().numpy(), want, rtol=RTOL, atol=ATOL)
        assert np.array_equal(a.cpu().numpy(), wk) and np.array_equal(b.cpu().numpy(), wv)
    logits = gemv.forward_qk(q, dk, new[0], *kp, T, SMIN, SMAX, bits=bits)
    lw = orc.forward_qk(case["q"][:, :, 0].numpy(), ok_, kn.numpy(), np_params(case["kp"]), T, bits, SMIN, SMAX)
    # half a unit of an fp16 logit on top of the stated tolerance
    np.testing.assert_allclose(logits.float().cpu().numpy(), lw, rtol=RTOL, atol=ATOL * max(1.0, np.abs(lw).max()))
    weights = torch.softmax(torch.from_numpy(lw).float() * 0.07 + mask[:, None], -1).half()
    out = gemv.forward_ov(weights.cuda(), dv, new[1], *vp, SMIN, SMAX, bits=bits)
    ow = orc.forward_ov(weights.double().numpy(), ov_, vn.numpy(), np_params(case["vp"]), bits, SMIN, SMAX)
    np.testing.assert_allclose(out.float().cpu().numpy(), ow, rtol=RTOL, atol=ATOL)
    assert np.array_equal(dk.cpu().numpy(), wk) and np.array_equal(dv.cpu().numpy(), wv)
    _status_ok()


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("G,T", EDGES)
def test_half_state(G, T, bits):
    test_gpu_half_state.test_fused_decode_against_numpy_restatement(2, 2 * G, 2, T, bits)


@pytest.mark.parametrize("B", [80, 160])      # forward_ov: two warps a stream up to 296 streams, one beyond
def test_ov_many_streams(B):
    T, Hkv, bits = 131, 2, 4
    g = torch.Generator().manual_seed(B)
    case = make_case(77, 1, Hkv, Hkv, T, bits)
    dk, dv, *_ = _prefill(case, T + 1)
    w = torch.softmax(torch.randn(B, Hkv, T + 1, generator=g), -1).half()
    vc = dv.expand(B, -1, -1, -1, -1, -1).contiguous()
    ov_ = dv.cpu().numpy()
    vn = case["v"][:, :, T]
    out = gemv.forward_ov(w.cuda(), vc, dev(vn).expand(B, -1, -1).contiguous()[:, :, None], *dev(case["vp"]), SMIN, SMAX, bits=bits)
    for b in (0, B // 2, B - 1):
        want = orc.forward_ov(w[b:b + 1].double().numpy(), ov_.copy(), vn.numpy(), np_params(case["vp"]), bits, SMIN, SMAX)
        np.testing.assert_allclose(out[b:b + 1].float().cpu().numpy(), want, rtol=RTOL, atol=ATOL)


# up to one stream per SM, one to two, two to eight, more: the lines at which tiles of 32 tokens begin
BY_SIZE = [(4, 1, 37, 64), (4, 1, 40, 64), (4, 1, 40, 65), (4, 1, 80, 65), (4, 2, 80, 255), (4, 2, 80, 256), (4, 4, 80, 64), (2, 1, 80, 64), (2, 1, 80, 65),
           (2, 2, 40, 255), (2, 4, 80, 255), (2, 4, 80, 256), (4, 1, 320, 64), (2, 4, 320, 130), (4, 8, 2, 511), (4, 8, 2, 512),
           (4, 8, 320, 1023), (4, 8, 320, 1024), (2, 8, 2, 255), (2, 8, 2, 256), (2, 8, 320, 191), (2, 8, 320, 192)]


@pytest.mark.parametrize("bits,G,n,T", BY_SIZE)
def test_tiles_by_size(bits, G, n, T):
    """Whole-head steps on either side of each line, canonical and contracted; n copies of two sequences."""
    B, Hkv = 2, 2
    case = make_case(1200 + T, B, G * Hkv, Hkv, T, bits)
    dk, dv, tk, tv, ok_, ov_, *_ = _prefill(case, T + 1)
    kn, vn = case["k"][:, :, T], case["v"][:, :, T]
    wk, wv = ok_.copy(), ov_.copy()
    want = orc.decode_attn(case["q"][:, :, 0].numpy(), wk, wv, kn.numpy(), vn.numpy(), np_params(case["kp"]), np_params(case["vp"]), T,
                           0.07, bits=bits, scale_min=SMIN, scale_max=SMAX)
    rep = lambda t: dev(t).repeat(n, *([1] * (t.dim() - 1)))
    for kw in (dict(k_tail=rep(tk), v_tail=rep(tv), tail_keep=True), dict()):
        a, b = rep(dk), rep(dv)
        got = gemv.decode_attn(rep(case["q"]), a, b, rep(kn[:, :, None]), rep(vn[:, :, None]), dev(case["kp"]), dev(case["vp"]), T, 0.07,
                               SMIN, SMAX, bits=bits, split_channels=False, **kw)
        np.testing.assert_allclose(got[:B].float().cpu().numpy(), want, rtol=RTOL, atol=ATOL)
        assert torch.equal(got, rep(got[:B])) and torch.equal(a, rep(a[:B])) and torch.equal(b, rep(b[:B]))
        assert np.array_equal(a[:B].cpu().numpy(), wk) and np.array_equal(b[:B].cpu().numpy(), wv)
    _status_ok()


SEGMENTS = [(2, 1, 256), (2, 2, 257), (4, 2, 300), (2, 1, 512), (4, 2, 513), (2, 4, 384), (2, 4, 385), (4, 4, 513)]


@pytest.mark.parametrize("bits,G,T", SEGMENTS)
def test_segments_by_size(bits, G, T):
    """Token segments at the lengths where their tiles change, with scale bounds that the tensor cores do not take."""
    B, Hkv = 2, 2
    case = make_case(1300 + T, B, G * Hkv, Hkv, T, bits)
    dk, dv, tk, tv, ok_, ov_, *_ = _prefill(case, T + 1, WIDE)
    kn, vn = case["k"][:, :, T], case["v"][:, :, T]
    want = orc.decode_attn(case["q"][:, :, 0].numpy(), ok_, ov_, kn.numpy(), vn.numpy(), np_params(case["kp"]), np_params(case["vp"]), T,
                           0.07, bits=bits, scale_min=WIDE[0], scale_max=WIDE[1])
    got = gemv.decode_attn(dev(case["q"]), dk, dv, dev(kn[:, :, None]), dev(vn[:, :, None]), dev(case["kp"]), dev(case["vp"]), T, 0.07,
                           *WIDE, bits=bits, k_tail=tk, v_tail=tv)
    np.testing.assert_allclose(got.float().cpu().numpy(), want, rtol=RTOL, atol=ATOL)
    assert np.array_equal(dk.cpu().numpy(), ok_) and np.array_equal(dv.cpu().numpy(), ov_)
    _status_ok()


@pytest.mark.parametrize("interval", [512, 544])
@pytest.mark.parametrize("bits", [4, 2])
def test_eight_heads_over_checkpoints(bits, interval):
    B, Hkv, G, T = 2, 2, 8, 1100
    case = make_case(1400, B, G * Hkv, Hkv, T, bits)
    ck = [gemv.alloc_ckpt(B, Hkv, 128, T + 1, interval, "cuda") for _ in range(2)]
    dk, dv, tk, tv, ok_, ov_, *_ = _prefill(case, T + 1, k_ckpt=ck[0], v_ckpt=ck[1], ckpt_interval=interval)
    kn, vn = case["k"][:, :, T], case["v"][:, :, T]
    want = orc.decode_attn(case["q"][:, :, 0].numpy(), ok_, ov_, kn.numpy(), vn.numpy(), np_params(case["kp"]), np_params(case["vp"]), T,
                           0.07, bits=bits, scale_min=SMIN, scale_max=SMAX)
    for kw in (dict(k_tail=tk, v_tail=tv, tail_keep=True), dict()):
        a, b = dk.clone(), dv.clone()
        got = gemv.decode_attn(dev(case["q"]), a, b, dev(kn[:, :, None]), dev(vn[:, :, None]), dev(case["kp"]), dev(case["vp"]), T, 0.07,
                               SMIN, SMAX, bits=bits, k_ckpt=ck[0], v_ckpt=ck[1], ckpt_interval=interval, **kw)
        np.testing.assert_allclose(got.float().cpu().numpy(), want, rtol=RTOL, atol=ATOL)
        assert np.array_equal(a.cpu().numpy(), ok_) and np.array_equal(b.cpu().numpy(), ov_)
    _status_ok()
