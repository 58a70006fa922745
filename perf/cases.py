"""The work a user has this library do, as measurable cases: packed-cache decode steps, prefills and appends.

Every case is one call (or the reference caller's sequence of calls) into ``adkv_b200.gemv`` on tensors that the
caller of an attention layer holds: packed caches, their five parameter tensors, tail states, queries and new tokens.
K, V, q and the parameters follow ``adkv_b200.synth`` (outlier channels, rotary embedding); caches are encoded from
them, so codes and scales are what decoding meets.  Head geometry, batches and context lengths come from the benchmark
workloads, the kernel benchmark's grid (batches 1-512, 128-2048 tokens, 32 heads x 128) and the tests.
"""
import math

import torch

from adkv_b200 import gemv, synth

D = 128
SMIN, SMAX = synth.SCALE_MIN, synth.SCALE_MAX


def listed():
    return [
        # one sequence just after a short prompt: the smallest step there is, nothing but latency and launches
        dict(name="decode_b1_t128", kind="decode", B=1, Hq=32, Hkv=32, T=128, bits=4, mask=False),
        # interactive serving: a handful of chats in mid-conversation, ragged length
        dict(name="decode_b4_t2047", kind="decode", B=4, Hq=32, Hkv=32, T=2047, bits=4, mask=False),
        # a left-padded batch through a model file: additive mask, odd length
        dict(name="decode_b24_t1531_mask", kind="decode", B=24, Hq=32, Hkv=32, T=1531, bits=4, mask=True),
        # the headline decode step: batch 128, 4096 cached tokens
        dict(name="decode_b128_t4096", kind="decode", B=128, Hq=32, Hkv=32, T=4096, bits=4, mask=False),
        # long context, grouped queries (32 query heads on 8 KV heads), 2-bit codes
        dict(name="decode_gqa_b32_t32768_2bit", kind="decode", B=32, Hq=32, Hkv=8, T=32768, bits=2, mask=False),
        # the same model with few sequences, on a cache that keeps state checkpoints
        dict(name="decode_gqa_b4_t16000_2bit_ckpt", kind="ckpt", B=4, Hq=32, Hkv=8, T=16000, bits=2, interval=512),
        # decoding caches that the reference's own kernels wrote (their fp16-state arithmetic)
        dict(name="decode_half_b64_t2048", kind="half", B=64, Hq=32, Hkv=32, T=2048, bits=4),
        # continuous batching: per-sequence lengths held on the device
        dict(name="decode_varlen_b48_t3000", kind="varlen", B=48, Hq=32, Hkv=32, T=3000, bits=4),
        # the reference's model file on top of this library: forward_qk, softmax in torch, forward_ov
        dict(name="qk_softmax_ov_b16_t1023", kind="trio", B=16, Hq=32, Hkv=32, T=1023, bits=4),
        # prefill of a batch of long prompts, K and V of one layer
        dict(name="prefill_b16_t8192", kind="prefill", B=16, Hkv=32, T=8192, bits=4),
        # prefill of one short prompt, 2-bit codes, ragged length
        dict(name="prefill_b1_t777_2bit", kind="prefill", B=1, Hkv=32, T=777, bits=2),
        # one token of every layer appended at once, after a prefill
        dict(name="append_32layers_b16_2bit", kind="append", B=16, Hkv=32, T=1023, bits=2, layers=32),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the ranges above; sizes over their logarithm, the product bounded by the listed maxima."""
    kind = rng.choice(["decode", "decode", "decode", "gqa", "ckpt", "half", "varlen", "trio", "prefill", "prefill", "append"])
    bits = rng.choice([4, 4, 2])
    if kind == "decode":
        B = _log(rng, 1, 128)
        return dict(kind="decode", B=B, Hq=32, Hkv=32, T=_log(rng, 100, 4096), bits=bits, mask=rng.random() < 0.3)
    if kind == "gqa":
        Hkv = rng.choice([8, 8, 16])
        T = _log(rng, 500, 32768)
        return dict(kind="decode", B=_log(rng, 1, max(1, min(64, 32 * 8 * 32768 // (Hkv * T)))), Hq=32, Hkv=Hkv, T=T,
                    bits=bits, mask=False)
    if kind == "ckpt":
        return dict(kind="ckpt", B=_log(rng, 1, 16), Hq=32, Hkv=rng.choice([8, 32]), T=_log(rng, 1000, 16000), bits=bits,
                    interval=rng.choice([256, 512, 1024]))
    if kind == "half":
        return dict(kind="half", B=_log(rng, 1, 64), Hq=32, Hkv=32, T=_log(rng, 100, 2048), bits=4)
    if kind == "varlen":
        return dict(kind="varlen", B=_log(rng, 2, 96), Hq=32, Hkv=rng.choice([32, 8]), T=_log(rng, 200, 3000), bits=bits)
    if kind == "trio":
        return dict(kind="trio", B=_log(rng, 1, 64), Hq=32, Hkv=32, T=_log(rng, 100, 2048), bits=4)
    if kind == "prefill":
        T = _log(rng, 50, 8192)
        return dict(kind="prefill", B=_log(rng, 1, 16), Hkv=rng.choice([32, 32, 8]), T=T, bits=bits)
    return dict(kind="append", B=_log(rng, 1, 16), Hkv=rng.choice([32, 8]), T=_log(rng, 100, 2000), bits=bits,
                layers=rng.choice([8, 16, 32]))


def _tokens(seed, B, H, T):
    """fp16 ``[B, H, T, 128]`` keys or values on the GPU, generated a few sequences at a time."""
    x = torch.empty(B, H, T, D, dtype=torch.float16, device="cuda")
    step = max(1, (1 << 28) // (H * T * D))
    for b in range(0, B, step):
        n = min(step, B - b)
        x[b:b + n] = synth.gen_kv(seed * 1009 + 17 * b, n, H, T, D, device="cuda")
    return x


def _filled(case, seed, T, half=False, ckpt=0):
    """Caches that hold ``T`` tokens, with room for one more, as a prefill leaves them."""
    B, H, bits = case["B"], case["Hkv"], case["bits"]
    kp, vp = synth.gen_params(seed + 3, H, D, bits, device="cuda"), synth.gen_params(seed + 4, H, D, bits, device="cuda")
    shape = (B, H, gemv.n_super_for(T + 1, bits), D // 4, 4, 4)
    kc, vc = (torch.zeros(shape, dtype=torch.uint8, device="cuda") for _ in range(2))
    st = dict(kp=kp, vp=vp, kc=kc, vc=vc)
    if not half:
        st["kt"], st["vt"] = (torch.zeros(B, H, 2, D, device="cuda") for _ in range(2))
    extra = {}
    if ckpt:
        st["kk"], st["vk"] = (gemv.alloc_ckpt(B, H, D, T + 1, ckpt, "cuda") for _ in range(2))
        extra = dict(k_ckpt=st["kk"], v_ckpt=st["vk"], ckpt_interval=ckpt)
    k, v = _tokens(2 * seed, B, H, T + 1), _tokens(2 * seed + 1, B, H, T + 1)
    gemv.encode_kv_pair(kc, k[:, :, :T], kp, vc, v[:, :, :T], vp, SMIN, SMAX, bits=bits, half_state=half,
                        k_tail=st.get("kt"), v_tail=st.get("vt"), **extra)
    st["k"], st["v"] = k[:, :, T:].contiguous(), v[:, :, T:].contiguous()
    if "Hq" in case:
        st["q"] = synth.gen_q(seed + 5, B, case["Hq"], D, device="cuda")
    return st


def prepare(case, seed):
    kind, B, H, T, bits = case["kind"], case["B"], case["Hkv"], case["T"], case["bits"]
    if kind == "prefill":
        st = dict(k=_tokens(2 * seed, B, H, T), v=_tokens(2 * seed + 1, B, H, T),
                  kp=synth.gen_params(seed + 3, H, D, bits, device="cuda"),
                  vp=synth.gen_params(seed + 4, H, D, bits, device="cuda"))
        shape = (B, H, gemv.n_super_for(T, bits), D // 4, 4, 4)
        st["kc"], st["vc"] = (torch.zeros(shape, dtype=torch.uint8, device="cuda") for _ in range(2))
        st["kt"], st["vt"] = (torch.zeros(B, H, 2, D, device="cuda") for _ in range(2))
    elif kind == "append":
        L = case["layers"]
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        shape = (L, B, H, gemv.n_super_for(T + 1, bits), D // 4, 4, 4)
        st = {n: torch.zeros(shape, dtype=torch.uint8, device="cuda") for n in ("kc", "vc")}
        for n in ("kt", "vt"):     # zero points around 0, scales around the size that standard-normal values settle at
            t = torch.randn(L, B, H, 2, D, generator=g, device="cuda")
            t[:, :, :, 1] = torch.exp(0.3 * t[:, :, :, 1] - 1.2)
            st[n] = t
        params = [[synth.gen_params(seed + 100 * i + j, H, D, bits, device="cuda") for j in range(2)] for i in range(L)]
        st["layers"] = gemv.LayerSet([(st["kc"][i], params[i][0], st["kt"][i], st["vc"][i], params[i][1], st["vt"][i])
                                      for i in range(L)], bits=bits)
        st["k"], st["v"] = (torch.randn(L, B, H, D, generator=g, device="cuda").half() for _ in range(2))
    else:
        st = _filled(case, seed, T, half=kind == "half", ckpt=case.get("interval", 0))
        if kind == "ckpt":
            n = gemv.decode_scratch_bytes(B, case["Hq"], H, T, case["interval"])
            st["scratch"] = torch.empty(n, dtype=torch.uint8, device="cuda")
        if kind == "varlen":       # lengths from a twentieth of the longest on; each tail is that of its own prefix
            g = torch.Generator().manual_seed(int(seed))
            lens = (T // 20 + torch.randint(0, T - T // 20 + 1, (B,), generator=g)).tolist()
            lens[0] = T
            st["lens"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
            k, v = _tokens(2 * seed, B, H, T + 1), _tokens(2 * seed + 1, B, H, T + 1)
            for b, n in enumerate(lens):
                gemv.encode_kv_pair(st["kc"][b:b + 1], k[b:b + 1, :, :n], st["kp"], st["vc"][b:b + 1], v[b:b + 1, :, :n],
                                    st["vp"], SMIN, SMAX, bits=bits, k_tail=st["kt"][b:b + 1], v_tail=st["vt"][b:b + 1])
        if case.get("mask"):       # left padding, as HF builds it: the lowest fp16 value on up to a third of the tokens
            g = torch.Generator().manual_seed(int(seed))
            pad = torch.randint(0, max(1, T // 3), (B,), generator=g)
            keep = torch.arange(T + 1)[None, :] >= pad[:, None]
            st["mask"] = torch.where(keep, 0.0, torch.finfo(torch.float16).min)[:, None, None, :].cuda()
    st["case"] = case
    return st


def run(st):
    """One pass.  ``tail_keep`` lets a decode step be repeated on the same cached tokens."""
    case = st["case"]
    kind, T, bits = case["kind"], case["T"], case["bits"]
    if kind == "prefill":
        gemv.encode_kv_pair(st["kc"], st["k"], st["kp"], st["vc"], st["v"], st["vp"], SMIN, SMAX, bits=bits,
                            k_tail=st["kt"], v_tail=st["vt"])
        return st["kc"], st["vc"], st["kt"], st["vt"]
    if kind == "append":
        gemv.append_kv_layers(st["layers"], st["k"], st["v"], T, SMIN, SMAX)
        return st["kc"], st["vc"], st["kt"], st["vt"]
    scaling = D ** -0.5
    if kind == "trio":
        logits = gemv.forward_qk(st["q"], st["kc"], st["k"], *st["kp"], T, SMIN, SMAX, bits=bits)
        weights = torch.softmax(logits.float() * scaling, dim=-1).to(torch.float16)
        out = gemv.forward_ov(weights, st["vc"], st["v"], *st["vp"], SMIN, SMAX, bits=bits)
        return logits, out, st["kc"], st["vc"]
    args = (st["q"], st["kc"], st["vc"], st["k"], st["v"], st["kp"], st["vp"])
    if kind == "varlen":
        out = gemv.decode_attn_varlen(*args, st["lens"], scaling, SMIN, SMAX, bits=bits, k_tail=st["kt"], v_tail=st["vt"],
                                      tail_keep=True)
    elif kind == "half":
        out = gemv.decode_attn(*args, T, scaling, SMIN, SMAX, bits=bits, half_state=True)
    elif kind == "ckpt":
        out = gemv.decode_attn(*args, T, scaling, SMIN, SMAX, bits=bits, k_tail=st["kt"], v_tail=st["vt"], tail_keep=True,
                               k_ckpt=st["kk"], v_ckpt=st["vk"], ckpt_interval=case["interval"], scratch=st["scratch"])
    else:
        out = gemv.decode_attn(*args, T, scaling, SMIN, SMAX, mask=st.get("mask"), bits=bits, k_tail=st["kt"],
                               v_tail=st["vt"], tail_keep=True)
    return out, st["kc"], st["vc"]


def work(case):
    """Bytes: packed codes, fp16 tokens, tails and results once each.  Operations: the recurrence is eight per code
    (five multiplies and adds for the state, three for the value); a query head adds a multiply-add per code of K and V."""
    B, H, T, bits = case["B"], case["Hkv"], case["T"], case["bits"]
    if case["kind"] == "varlen":
        T = (T + T // 20) / 2
    row = 2 * B * H * D                                    # one token of K and V, elements
    codes = row * T
    if case["kind"] == "prefill":
        return dict(bytes=codes * (2 + bits / 8) + row * 8, flops=12 * codes)
    if case["kind"] == "append":
        return dict(bytes=case["layers"] * row * (2 + 16 + 8), flops=12 * row * case["layers"])
    Hq = case["Hq"]
    b = codes * bits / 8 + row * 2 + 2 * B * Hq * D * 2    # caches, new tokens, q and output
    if case["kind"] == "ckpt":
        b += row * 8 * (T // case["interval"])
    elif case["kind"] == "trio":
        b += 4 * B * Hq * (T + 1) * 2                      # logits and weights, written and read
    if case["kind"] not in ("half", "trio"):
        b += row * 8                                       # tail states
    return dict(bytes=b, flops=codes * (8 + 2 * Hq / H))


def tolerance(case):
    """About four times what was measured on these inputs.  A fused step against the same step in 64 bits: rel 2.1e-4,
    max 4.7e-4 (half an fp16 unit of the output).  The three-call sequence rounds logits and weights to fp16 in between:
    1.4e-3 and 1.3e-2 against 64 bits.  The fp16-state arithmetic adds its products in fp16: fused against three calls
    1.7e-3 and 1.6e-2.  Packed codes, appended codes and tail states are defined bit for bit."""
    kind = case["kind"]
    if kind in ("prefill", "append"):
        return "exact"
    if kind == "half":
        return dict(rel=7e-3, max=6.5e-2)
    if kind == "trio":
        return dict(rel=6e-3, max=5e-2)
    return dict(rel=8e-4, max=2.5e-3)
