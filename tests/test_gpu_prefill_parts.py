"""Prefills whose CTAs do not come out even on the SMs run as two launches side by side: bytes, states and checkpoints are those of the
one-stream call, whatever follows on the stream sees both parts, and the pair can be captured.  Needs a B200."""
import pytest
import torch

from adkv_b200 import gemv
from oracle import adkv_oracle as orc
from tests.util import SMAX, SMIN, dev, make_case

pytestmark = pytest.mark.gpu


def _prefill(case, n, H, T, bits, interval, start):
    rep = lambda t: dev(t).repeat(n, 1, 1, 1)
    kc = torch.zeros(orc.cache_shape(n, H, orc.n_super_for(T, bits), 128), dtype=torch.uint8, device="cuda")
    vc, kt, vt = torch.zeros_like(kc), torch.zeros(n, H, 2, 128, device="cuda"), torch.zeros(n, H, 2, 128, device="cuda")
    extra = {}
    if interval:
        extra = dict(k_ckpt=gemv.alloc_ckpt(n, H, 128, T, interval, "cuda"), v_ckpt=gemv.alloc_ckpt(n, H, 128, T, interval, "cuda"),
                     ckpt_interval=interval)
    kp, vp = dev(case["kp"]), dev(case["vp"])
    chunks = [(0, start), (start, T)] if start else [(0, T)]
    x = [(rep(case["k"][:, :, lo:hi]), rep(case["v"][:, :, lo:hi])) for lo, hi in chunks]

    def run():
        for (lo, hi), (k, v) in zip(chunks, x):
            gemv.encode_kv_pair(kc, k, kp, vc, v, vp, SMIN, SMAX, bits=bits, t_start=lo, k_tail=kt, v_tail=vt, **extra)
        return [t.clone() for t in (kc, vc, kt, vt, *(extra[n] for n in ("k_ckpt", "v_ckpt") if extra))]
    return run, (kc, vc, kt, vt)


# 600, 740, 890, 1036 and 1224 slices leave 8, 148, 2, 148 and 40 over an even number on 148 SMs; 742 leaves 150 and stays one launch, as do
# 740 slices of 2-bit codes below 2048 tokens and 1036 below 384
SHAPES = [(60, 5, 256, 4, 0, 0), (74, 5, 259, 2, 0, 0), (89, 5, 300, 4, 128, 0), (74, 7, 405, 2, 96, 0), (74, 7, 305, 2, 96, 0), (74, 5, 600, 4, 0, 331),
          (53, 7, 260, 4, 0, 0), (102, 6, 259, 2, 0, 0), (37, 10, 2050, 2, 0, 0)]


@pytest.mark.parametrize("B,H,T,bits,interval,start", SHAPES)
def test_parts_of_a_prefill(B, H, T, bits, interval, start):
    case = make_case(2000 + T, 1, H, H, T, bits)
    many, one = (_prefill(case, n, H, T, bits, interval, start)[0]() for n in (B, 1))
    assert gemv.device_status() == 0
    for m, o in zip(many, one):
        m, o = m.view(torch.uint8), o.view(torch.uint8)
        assert torch.equal(m, o.repeat(B, *([1] * (o.dim() - 1))))


def test_parts_captured():
    B, H, T, bits = 74, 5, 270, 4
    case = make_case(2100, 1, H, H, T, bits)
    run, bufs = _prefill(case, B, H, T, bits, 0, 0)
    want = run()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        got = run()
    for t in bufs:
        t.zero_()
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(got, want))
    assert gemv.device_status() == 0
