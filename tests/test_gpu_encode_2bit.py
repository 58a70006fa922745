"""2-bit prefill of few streams (codes from comparisons) against exact fp32 division in numpy and against the quotient form that
launches with many streams take, bit for bit.  Needs a B200."""
import numpy as np
import pytest
import torch

from adkv_b200 import gemv, synth
from oracle import adkv_oracle as orc
from tests.util import SMAX, SMIN, np_params

pytestmark = pytest.mark.gpu

H, D, MANY = 2, 128, 160     # 160 sequences x 2 heads x K and V: 640 streams, well past the 444 that count as few


def _inputs(T, special):
    g = torch.Generator().manual_seed(T)
    p = [t.clone() for t in synth.gen_params(5, H, D, 2)]
    x = torch.randn(1, H, T, D, generator=g)
    x[..., ::9] *= 20
    # frozen states: quotients that are multiples of a half, and the fp16 numbers next to them
    p[2][:, ::4] = 0
    p[3][:, ::4] = 0
    p[1][:, ::4] = torch.rand(H, D // 4, generator=g).half() * 2 + 0.1
    k = torch.randint(-5, 6, (1, H, T, D // 4), generator=g) * 0.5
    near = (p[1][:, None, ::4].float() * k).half().contiguous()
    step = torch.randint(-1, 2, near.shape, generator=g).to(torch.int16)
    x = x.half()
    x[..., ::4] = torch.where(near == 0, near, (near.view(torch.int16) + step).view(torch.float16))
    p[4][:, 3::16] = 100.0       # scales that rest at the lower bound
    if special:
        x[0, 0, ::3, 1] = float("nan")
        x[0, 0, ::5, 2] = float("inf")
        x[0, 1, ::5, 2] = -float("inf")
        p[0][:, 5] = -0.0        # zero points of -0, moved by nothing while the codes are 0
        x[..., 5] = 0.0
        p[2][0, 6] = float("inf")
        p[3][:, 7] = 60.0        # scales from one bound to the other within a token
        p[1][:, 10] = 0.0        # initial scale under the eps guard
    return x, tuple(p)


def _encode(x, p, B, smin, smax, t_start=0):
    xs = x.cuda().expand(B, -1, -1, -1).contiguous()
    T = x.shape[2]
    pc = tuple(t.cuda() for t in p)
    kc, vc = (torch.zeros(B, H, gemv.n_super_for(T, 2), D // 4, 4, 4, dtype=torch.uint8, device="cuda") for _ in range(2))
    kt, vt = (torch.zeros(B, H, 2, D, device="cuda") for _ in range(2))
    for a, b in ((0, t_start), (t_start, T)):
        if a < b:
            gemv.encode_kv_pair(kc, xs[:, :, a:b], pc, vc, xs[:, :, a:b], pc, smin, smax, bits=2, k_tail=kt, v_tail=vt, t_start=a)
    assert torch.equal(kc, vc) and torch.equal(kt.view(torch.int32), vt.view(torch.int32))
    return kc, kt


def _reference(x, p, smin, smax, state=None):
    """Codes and final state by numpy's fp32 division; minimum and maximum as on the device, where a NaN gives the other operand."""
    zp, s, alpha, beta, target = (np.broadcast_to(a.astype(np.float32), (1, H, D)) for a in np_params(p))
    if state is not None:
        zp, s = state
    lo, hi = np.float32(smin), np.float32(smax)
    codes = np.empty(x.shape, np.int8)
    with np.errstate(all="ignore"):
        for t in range(x.shape[2]):
            ss = np.fmax(s, np.float32(1e-8))
            q = np.fmin(np.fmax(np.rint((x[:, :, t] - zp) / ss), np.float32(-2)), np.float32(1))
            codes[:, :, t] = q.astype(np.int8)
            zp = zp + alpha * (q * ss)
            s = np.fmin(np.fmax(s + s * beta * (np.abs(q) - target), lo), hi)
    return codes, np.stack([zp, s], axis=2)


@pytest.mark.parametrize("T,t_start", [(7, 0), (8, 0), (9, 0), (16, 0), (33, 0), (777, 0), (100, 13)])
@pytest.mark.parametrize("special,smin,smax", [(False, SMIN, SMAX), (True, SMIN, SMAX), (True, 0.0, 1e30)])
def test_few_streams(T, t_start, special, smin, smax):
    x, p = _inputs(T, special)
    kc, kt = _encode(x, p, 1, smin, smax, t_start)
    mc, mt = _encode(x, p, MANY, smin, smax, t_start)
    assert torch.equal(kc[0], mc[0]) and torch.equal(mc[0], mc[MANY - 1])
    assert torch.equal(kt[0].view(torch.int32), mt[0].view(torch.int32))
    codes, tail = _reference(x.float().numpy(), p, smin, smax)
    assert np.array_equal(kc.cpu().numpy(), orc.pack_codes(codes, 2, kc.shape[2]))
    assert np.array_equal(kt.cpu().numpy(), tail, equal_nan=True)
    if not special:
        want = np.zeros(kc.shape, np.uint8)
        orc.encode_kv(want, x.numpy(), np_params(p), 2, smin, smax)
        assert np.array_equal(kc.cpu().numpy(), want)


def test_scale_overflows_within_a_group():
    """Without an upper bound a scale may grow from 3e28 to 2e38 within eight tokens: twice the scale overflows, and the zero point
    with it, although alpha is 0."""
    T = 8
    p = [t.clone() for t in synth.gen_params(5, H, D, 2)]
    p[2][:], p[3][:], p[4][:] = 0.0, 12.0, 0.0
    x = torch.randn(1, H, T, D, generator=torch.Generator().manual_seed(1)).half()
    start = [np.full((1, H, D), v, np.float32) for v in (3.3e38, 3.113e28)]
    codes, tail = _reference(x.float().numpy(), tuple(p), 0.0, np.inf, start)
    assert np.isnan(tail[:, :, 0]).all() and codes[:, :, -1].max() == -2
    pc = tuple(t.cuda() for t in p)
    kc, vc = (torch.zeros(1, H, 1, D // 4, 4, 4, dtype=torch.uint8, device="cuda") for _ in range(2))
    kt, vt = (torch.from_numpy(np.stack(start, axis=2)).cuda() for _ in range(2))
    gemv.encode_kv_pair(kc, x.cuda(), pc, vc, x.cuda(), pc, 0.0, float("inf"), bits=2, k_tail=kt, v_tail=vt, t_start=8)
    assert np.array_equal(orc.unpack_codes(kc.cpu().numpy(), 16, 2)[:, :, 8:], codes)
    assert np.array_equal(kt.cpu().numpy(), tail, equal_nan=True) and np.array_equal(vt.cpu().numpy(), tail, equal_nan=True)
