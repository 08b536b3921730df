"""The work that users have this framework do, as cases that can be timed and compared.

Every case goes through the public entry points of ``rustorch_b200`` the way a user's program calls them.  Six kinds:

    decode_step  one layer's step of a token loop: rope_kv_append, then gqa_decode on the cache it wrote to
    decode       attention of a batch of single-token queries against a KV cache (gqa_decode)
    prefill      device-resident bf16 forward (prefill_bf16): whole prompts, padded batches, prompt chunks on a cache
    mha          activations in the modules' own [B, T, H*hd] layout (mha_prefill_bf16)
    train_bf16, train_f32   forward and backward of a training step on device tensors
    host         the drop-in call on host f32 arrays (flash_forward_masked)

Inputs are N(0, 1) as in the headline configurations (a layer norm keeps Q, K and V near that in real models).
Ragged lengths are spread evenly over [lo, hi] and dealt to the sequences in an order that the seed picks, so the
amount of work is a property of the case and not of the seed.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import rustorch_b200 as rt

# ------------------------------------------------------------------------------------------------ the cases


def listed():
    return [
        # one user of a Llama-like model with 8 KV heads: a layer's step at about a thousand tokens of context
        dict(name="decode_step_1seq", kind="decode_step", B=1, Hq=32, Hkv=8, D=128, max_seq=4096, lo=1000, hi=1000),
        # a small batch on a model of head dim 256, lengths that are multiples of nothing
        dict(name="decode_7seq_d256", kind="decode", B=7, Hq=16, Hkv=2, D=256, max_seq=3000, lo=100, hi=3000),
        # a full server: 64 sequences of 1024 to 8192 tokens
        dict(name="decode_64seq", kind="decode", B=64, Hq=32, Hkv=8, D=128, max_seq=8192, lo=1024, hi=8192),
        # one GPU's eighth of a million-token context
        dict(name="decode_long_context", kind="decode", B=1, Hq=32, Hkv=8, D=128, max_seq=131072, lo=131072, hi=131072),
        # the small causal forward that the CPU reference is quoted on
        dict(name="prefill_small", kind="prefill", B=1, Hq=8, Hkv=8, Nq=2048, Nkv=2048, D=64, causal=True, lo=0, hi=0),
        # Llama-7B-like prompts
        dict(name="prefill_large", kind="prefill", B=4, Hq=32, Hkv=32, Nq=4096, Nkv=4096, D=128, causal=True, lo=0, hi=0),
        # a padded batch: 16 sequences of 256 to 2048 valid keys, causal as well
        dict(name="prefill_padded", kind="prefill", B=16, Hq=16, Hkv=16, Nq=2048, Nkv=2048, D=64, causal=True, lo=256,
             hi=2048),
        # a chunk of a long prompt against the cache of what came before it
        dict(name="prefill_chunk", kind="prefill", B=1, Hq=32, Hkv=8, Nq=500, Nkv=8192, D=128, causal=True, lo=6001,
             hi=6001),
        # an encoder layer: no causal mask, keys of padding tokens left out
        dict(name="mha_encoder", kind="mha", B=8, T=777, H=12, Hkv=12, D=64, causal=False, keep=True),
        # a training step of a decoder layer
        dict(name="train_bf16", kind="train_bf16", B=4, H=32, N=2048, D=128, causal=True),
        # the same in exact f32, at the sizes where people check their models in it
        dict(name="train_f32", kind="train_f32", B=2, H=8, N=1000, D=64, causal=True),
        # the reference's own call: host f32 slices in, host f32 slice out, its default precision
        dict(name="host_f32", kind="host", B=1, H=8, N=2048, D=64, mask="causal", precision="f32"),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    """Evenly over the logarithm, every integer possible."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# (query heads, KV heads): no grouping, and groups of 2, 4 and 8
_HEADS = [(8, 8), (16, 16), (32, 32), (12, 12), (16, 8), (32, 8), (32, 16), (16, 2), (24, 6), (64, 8)]


def _draw_once(rng: random.Random) -> dict:
    kind = rng.choice(["decode_step", "decode", "decode", "prefill", "prefill", "prefill", "mha", "train_bf16",
                       "train_f32", "host"])
    Hq, Hkv = rng.choice(_HEADS)
    if kind in ("decode_step", "decode"):
        D = rng.choice([64, 128, 128, 256])
        B = _log_int(rng, 1, 16 if kind == "decode_step" else 64)
        max_seq = _log_int(rng, 512, 131072)
        hi = rng.randint(max(1, max_seq // 2), max_seq)
        lo = hi if B == 1 else rng.randint(max(1, hi // 8), hi)
        return dict(kind=kind, B=B, Hq=Hq, Hkv=Hkv, D=D, max_seq=max_seq, lo=lo, hi=hi)
    if kind == "prefill":
        B, D, Nq = _log_int(rng, 1, 16), rng.choice([64, 128]), _log_int(rng, 32, 4096)
        what = rng.choice(["whole", "whole", "padded", "chunk"])
        if what == "whole":
            return dict(kind=kind, B=B, Hq=Hq, Hkv=Hkv, Nq=Nq, Nkv=Nq, D=D, causal=rng.random() < 0.75, lo=0, hi=0)
        if what == "padded":
            return dict(kind=kind, B=B, Hq=Hq, Hkv=Hkv, Nq=Nq, Nkv=Nq, D=D, causal=True, lo=max(1, Nq // 8), hi=Nq)
        Nq, max_seq = _log_int(rng, 32, 1024), _log_int(rng, 1024, 16384)
        return dict(kind=kind, B=min(B, 4), Hq=Hq, Hkv=Hkv, Nq=Nq, Nkv=max_seq, D=D, causal=True,
                    lo=max(Nq, max_seq // 4), hi=max_seq)
    if kind == "mha":
        causal = rng.random() < 0.5
        return dict(kind=kind, B=_log_int(rng, 1, 16), T=_log_int(rng, 32, 2048), H=Hq, Hkv=Hkv, D=rng.choice([64, 128]),
                    causal=causal, keep=not causal and rng.random() < 0.5)
    if kind == "train_bf16":
        return dict(kind=kind, B=_log_int(rng, 1, 8), H=Hq, N=_log_int(rng, 128, 4096), D=rng.choice([64, 128]),
                    causal=rng.random() < 0.75)
    if kind == "train_f32":
        return dict(kind=kind, B=_log_int(rng, 1, 4), H=rng.choice([4, 8, 12, 16]), N=_log_int(rng, 64, 1500),
                    D=rng.choice([32, 64, 80, 128]), causal=rng.random() < 0.75)
    precision = rng.choice(["f32", "f32", "bf16"])
    return dict(kind=kind, B=_log_int(rng, 1, 4), H=rng.choice([4, 8, 12, 16]), N=_log_int(rng, 64, 2500),
                D=rng.choice([64, 128]) if precision == "bf16" else rng.choice([32, 64, 80, 128]),
                mask=rng.choice(["none", "causal", "causal", "padding"]), precision=precision)


# the largest that a case of a kind may be, (bytes, flops): its listed case, or what the largest listed case of all
# takes about as long as
_MOST = {"decode_step": (1.2e9, 1e15), "decode": (1.2e9, 1e15), "prefill": (1e15, 0.55e12), "mha": (1e15, 0.3e12),
         "train_bf16": (1e15, 0.5e12), "train_f32": (1e15, 12e9), "host": (40e6, 12e9)}


def draw(rng):
    while True:
        case = _draw_once(rng)
        w, most = work(case), _MOST[case["kind"]]
        caches = case["B"] * case.get("Hkv", 1) * case.get("max_seq", 1) * case["D"] * 4
        if w["bytes"] <= most[0] and w["flops"] <= most[1] and caches <= 4 << 30:
            return case


# ------------------------------------------------------------------------------------------------ inputs


def _spread(B: int, lo: int, hi: int):
    return [lo + int(round((hi - lo) * (i + 0.5) / B)) for i in range(B)]


def _lens(case, seed):
    lens = _spread(case["B"], case["lo"], case["hi"])
    random.Random(seed).shuffle(lens)
    return lens


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape, dtype=torch.bfloat16):
        return torch.randn(shape, dtype=dtype, device="cuda", generator=g)

    kind, B, D = case["kind"], case["B"], case["D"]
    s = {"case": case}
    if kind in ("decode_step", "decode"):
        Hq, Hkv, S = case["Hq"], case["Hkv"], case["max_seq"]
        lens = _lens(case, seed)
        s.update(q=randn(B, Hq, D), k_cache=randn(B, Hkv, S, D), v_cache=randn(B, Hkv, S, D))
        if kind == "decode_step":
            # the token loop's own buffers: the output is reused from step to step, as are the position counters
            s.update(k_in=randn(B, Hkv, D), v_in=randn(B, Hkv, D), inv_freq=rt.rope_inv_freq(D),
                     out=torch.empty((B, Hq, D), dtype=torch.bfloat16, device="cuda"))
            if B == 1:
                s.update(pos=lens[0] - 1, kv_len=lens[0])
            else:
                s.update(positions=_i32([n - 1 for n in lens]), kv_lens=_i32(lens))
        elif B == 1:
            s.update(kv_len=lens[0])
        else:
            s.update(kv_lens=_i32(lens))
    elif kind == "prefill":
        Hq, Hkv, Nq, Nkv = case["Hq"], case["Hkv"], case["Nq"], case["Nkv"]
        s.update(q=randn(B, Hq, Nq, D), k=randn(B, Hkv, Nkv, D), v=randn(B, Hkv, Nkv, D), options={})
        if case["hi"]:
            lens = _lens(case, seed)
            s["options"]["kv_lens"] = _i32(lens)
            if Nkv != Nq:  # the chunk's queries are the last Nq of the visible positions
                s["options"]["q_offsets"] = _i32([n - Nq for n in lens])
    elif kind == "mha":
        T, H, Hkv = case["T"], case["H"], case["Hkv"]
        s.update(q=randn(B, T, H * D), k=randn(B, T, Hkv * D), v=randn(B, T, Hkv * D), options={})
        if case["keep"]:  # the tail of every sequence is padding, between none and half of it
            first_pad = _spread(B, T // 2, T)
            random.Random(seed).shuffle(first_pad)
            s["options"]["key_keep"] = torch.arange(T, device="cuda")[None, :] < _i32(first_pad)[:, None]
    elif kind in ("train_bf16", "train_f32"):
        dtype = torch.bfloat16 if kind == "train_bf16" else torch.float32
        s.update({n: randn(B, case["H"], case["N"], D, dtype=dtype) for n in ("q", "k", "v", "d_out")})
    else:
        r = np.random.default_rng(seed)
        H, N = case["H"], case["N"]
        q, k, v = (r.standard_normal(B * H * N * D, dtype=np.float32) for _ in range(3))
        mask = {"none": rt.Mask.none, "causal": rt.Mask.causal,
                "padding": lambda: rt.Mask.padding(np.arange(N) < N - N // 4)}[case["mask"]]()
        s.update(shape=rt.AttentionShape.new(B, H, N, D), q=q, k=k, v=v, mask=mask, out=np.empty_like(q))
    return s


# ------------------------------------------------------------------------------------------------ one pass


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode_step":
        rt.rope_kv_append(s["q"], s["k_in"], s["v_in"], s["k_cache"], s["v_cache"], s["inv_freq"], pos=s.get("pos"),
                          positions=s.get("positions"))
        out, _ = rt.gqa_decode(s["q"], s["k_cache"], s["v_cache"], kv_lens=s.get("kv_lens"), kv_len=s.get("kv_len"),
                               out=s["out"], return_lse=False)
        return {"out": out, "q": s["q"], "k_cache": s["k_cache"], "v_cache": s["v_cache"]}
    if kind == "decode":
        return rt.gqa_decode(s["q"], s["k_cache"], s["v_cache"], kv_lens=s.get("kv_lens"), kv_len=s.get("kv_len"))
    if kind == "prefill":
        return rt.prefill_bf16(s["q"], s["k"], s["v"], causal=case["causal"], **s["options"])
    if kind == "mha":
        return rt.mha_prefill_bf16(s["q"], s["k"], s["v"], case["H"], case["Hkv"], causal=case["causal"], **s["options"])
    if kind in ("train_bf16", "train_f32"):
        forward, backward = ((rt.prefill_bf16, rt.backward_bf16) if kind == "train_bf16" else
                             (rt.prefill_f32, rt.backward_f32))
        out, lse = forward(s["q"], s["k"], s["v"], causal=case["causal"])
        dq, dk, dv = backward(s["q"], s["k"], s["v"], out, s["d_out"], lse, causal=case["causal"])
        return {"out": out, "lse": lse, "dq": dq, "dk": dk, "dv": dv}
    rt.flash_forward_masked(s["shape"], s["q"], s["k"], s["v"], s["mask"], s["out"], case["precision"])
    return s["out"]


# ------------------------------------------------------------------------------------------------ what a pass needs


def _pairs(case) -> float:
    """(query, key) pairs of one head that no mask hides, over the batch."""
    kind, B = case["kind"], case["B"]
    if kind == "prefill":
        Nq, Nkv = case["Nq"], case["Nkv"]
        lens = _spread(B, case["lo"], case["hi"]) if case["hi"] else [Nkv] * B
        total = 0.0
        for n in lens:
            off = n - Nq if Nkv != Nq else 0  # row i sees min(n, i + 1 + off) keys
            if not case["causal"]:
                total += Nq * n
            else:
                m = min(Nq, n - off)
                total += m * off + m * (m + 1) / 2 + (Nq - m) * n
        return total
    N = case["T"] if kind == "mha" else case["N"]
    if kind == "mha" and case["keep"]:
        return float(sum(N * n for n in _spread(B, N // 2, N)))
    if kind == "host" and case["mask"] == "padding":
        return float(B * N * (N - N // 4))
    causal = case["mask"] == "causal" if kind == "host" else case["causal"]
    return B * (N * (N + 1) / 2.0 if causal else float(N) * N)


def work(case):
    kind, B, D = case["kind"], case["B"], case["D"]
    if kind in ("decode_step", "decode"):
        Hq, Hkv = case["Hq"], case["Hkv"]
        tokens = sum(_spread(B, case["lo"], case["hi"]))
        b = tokens * Hkv * D * 4 + B * Hq * D * 4
        b += B * (Hq + 3 * Hkv) * D * 2 if kind == "decode_step" else B * Hq * 4
        return {"bytes": b, "flops": 4.0 * tokens * Hq * D}
    if kind == "prefill":
        keys = sum(_spread(B, case["lo"], case["hi"])) if case["hi"] else B * case["Nkv"]
        rows = B * case["Hq"] * case["Nq"]
        return {"bytes": rows * (D * 4 + 4) + keys * case["Hkv"] * D * 4, "flops": 4.0 * D * case["Hq"] * _pairs(case)}
    if kind == "mha":
        return {"bytes": B * case["T"] * (case["H"] * (D * 4 + 4) + case["Hkv"] * D * 4),
                "flops": 4.0 * D * case["H"] * _pairs(case)}
    n = B * case["H"] * case["N"]
    if kind == "host":
        return {"bytes": n * D * 16, "flops": 4.0 * D * case["H"] * _pairs(case)}
    size = 2 if kind == "train_bf16" else 4
    # q, k, v, d_out in; out and lse out; three f32 gradients out.  Two products forward, five backward.
    return {"bytes": n * (D * (5 * size + 12) + 4), "flops": 14.0 * D * case["H"] * _pairs(case)}


def tolerance(case):
    if case["kind"] == "train_f32" or case.get("precision") == "f32":
        return {"rel": 1e-5, "max": 5e-4}  # sums of up to a few thousand f32 terms, one exponential each
    if case["kind"] == "train_bf16":
        return {"rel": 1e-2}  # P and dS are rounded to bf16 between the products
    return {"rel": 5e-3, "max": 0.1}  # P and the output are rounded to bf16
