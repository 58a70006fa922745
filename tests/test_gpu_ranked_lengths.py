"""Device-side lengths taken longest first: what a sequence gets does not depend on the order.  Needs a B200."""
import pytest
import torch

from adkv_b200 import gemv, synth
from tests.util import SMAX, SMIN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hkv,cap,room", [(2, 80, 520, 520), (50, 3, 512, 512), (65, 3, 512, 512), (128, 2, 512, 512),
                                            (129, 2, 512, 512), (60, 3, 512, 4000), (60, 3, 513, 4000)])
def test_ranked_lengths(B, Hkv, cap, room):
    """More than 148 streams, 512 tokens and more: up to 128 sequences are ranked, unless all are shorter.  Equal lengths, empty
    sequences and full caches among them; every sequence as the dense call with one warp per tensor gives it (the same scan:
    bit-equal)."""
    D, bits = 128, 4
    g = torch.Generator().manual_seed(B)
    lens = torch.randint(0, cap, (B,), generator=g)
    lens[::7] = lens[0]
    lens[1], lens[B - 1] = 0, cap - 1
    kp, vp = synth.gen_params(3, Hkv, D, bits, device="cuda"), synth.gen_params(4, Hkv, D, bits, device="cuda")
    shape = (B, Hkv, gemv.n_super_for(room, bits), D // 4, 4, 4)
    kc, vc = (torch.randint(0, 256, shape, dtype=torch.uint8, generator=g).cuda() for _ in range(2))
    kt, vt = (torch.rand(B, Hkv, 2, D, generator=g).cuda() + 0.1 for _ in range(2))
    q, kn, vn = (torch.randn(B, Hkv, 1, D, generator=g).half().cuda() for _ in range(3))
    refs = [x.clone() for x in (kc, vc, kt, vt)]
    got = gemv.decode_attn_varlen(q, kc, vc, kn, vn, kp, vp, lens.int().cuda(), 0.05, SMIN, SMAX, bits=bits, k_tail=kt, v_tail=vt)
    want = torch.empty_like(got)
    for b, T in enumerate(lens.tolist()):
        one = slice(b, b + 1)
        want[one] = gemv.decode_attn(q[one], refs[0][one], refs[1][one], kn[one], vn[one], kp, vp, T, 0.05, SMIN, SMAX, bits=bits,
                                     k_tail=refs[2][one], v_tail=refs[3][one], split_channels=False)
    assert gemv.device_status() == 0
    assert torch.equal(got, want)
    for a, b in zip((kc, vc, kt, vt), refs):
        assert torch.equal(a, b)
