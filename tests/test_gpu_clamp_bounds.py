"""Scale bounds that are unusual but accepted: a scale_max below the eps of the quantiser, and below scale_min.  Needs a B200."""
import numpy as np
import pytest
import torch

from adkv_b200 import gemv, synth
from oracle import adkv_oracle as orc
from tests.util import np_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("smin,smax", [(0.02, 1e-9), (1e-9, 2e-9), (0.02, 0.01)])
@pytest.mark.parametrize("bits,G", [(4, 1), (2, 1), (4, 4)])
def test_upper_bound_below_eps(bits, G, smin, smax):
    """The upper bound is applied last, so scales rest at smax; the eps guard then still decides what a code is worth.  Zero
    points that move by 60000 times that make it visible in fp16.  Relative tolerance: an fp16 result is within 2^-11, the
    contracted replay of 75 tokens within 75 * 2^-22."""
    B, Hkv, T, D = 1, 2, 75, 128
    g = torch.Generator().manual_seed(bits + G)
    p = list(synth.gen_params(1, Hkv, D, bits))
    p[2] = torch.full((Hkv, D), 60000.0 if smax < 1e-8 else 0.05).half()
    p[1] = torch.full((Hkv, D), 1e-7).half()
    p = tuple(p)
    kc, vc = (torch.randint(0, 256, (B, Hkv, gemv.n_super_for(T + 33, bits), D // 4, 4, 4), dtype=torch.uint8, generator=g) for _ in range(2))
    q, kn, vn = (torch.randn(B, h, 1, D, generator=g).half() for h in (G * Hkv, Hkv, Hkv))
    ck = [gemv.alloc_ckpt(B, Hkv, D, T + 1, 128, "cuda") for _ in range(2)]
    wk, wv = kc.numpy().copy(), vc.numpy().copy()
    want = orc.decode_attn(q[:, :, 0].numpy(), wk, wv, kn[:, :, 0].numpy(), vn[:, :, 0].numpy(), np_params(p), np_params(p), T, 0.5,
                           bits=bits, scale_min=smin, scale_max=smax)
    pc = tuple(t.cuda() for t in p)
    for kw in (dict(split_channels=False, fast=False), dict(split_channels=False, fast=True), dict(split_channels=True, fast=False),
               dict(k_ckpt=ck[0], v_ckpt=ck[1], ckpt_interval=128, fast=False)):
        a, b = kc.cuda(), vc.cuda()
        got = gemv.decode_attn(q.cuda(), a, b, kn.cuda(), vn.cuda(), pc, pc, T, 0.5, smin, smax, bits=bits, **kw)
        err = np.linalg.norm(got.float().cpu().numpy() - want) / np.linalg.norm(want)
        assert err < 1e-3, (kw, err)
        if not kw["fast"]:
            assert np.array_equal(a.cpu().numpy(), wk) and np.array_equal(b.cpu().numpy(), wv), kw
    lw = orc.forward_qk(q[:, :, 0].numpy(), kc.numpy().copy(), kn[:, :, 0].numpy(), np_params(p), T, bits, smin, smax)
    logits = gemv.forward_qk(q.cuda(), kc.cuda(), kn.cuda(), *pc, T, smin, smax, bits=bits)
    assert np.linalg.norm(logits.float().cpu().numpy() - lw) < 1e-3 * np.linalg.norm(lw)
    assert gemv.device_status() == 0
