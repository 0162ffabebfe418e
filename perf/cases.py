"""The workloads whose speed this library is judged by: dense attention through its public Python entry points.

Two kinds of pass, as user programs make them:

* ``forward``: ``flash_attn2_b200.fwd`` without gradients, which returns the output and the LSE. Prefill (as many
  queries as keys), chunked prefill (a chunk of queries against a longer K/V cache) and decode (one or a few queries
  against the filled part of a preallocated cache).
* ``train``: ``flash_attn2_b200.flash_attn_func`` and its gradients, through autograd.

Packed batches (``flash_attn_varlen_func``) are not timed here: a forward of a large packed batch, run in a loop with
other kernels, once ended in a launch failure whose cause was never shown, so that path is not looped on a GPU.

The inputs are N(0, 1), the convention of the benchmark and of the tests.
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "kernels-community-rs_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import flash_attn2_b200 as fa2  # noqa: E402

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _case(**kw):
    case = {"kind": "forward", "batch": 1, "heads": 16, "heads_k": 16, "seqlen_q": 128, "seqlen_k": 128, "head_dim": 128,
            "dtype": "bf16", "causal": False, "window": -1, "softcap": 0.0, "alibi": False, "deterministic": False,
            "layout": "separate"}
    case.update(kw)
    return case


def listed():
    return [
        # The smallest call: one short sequence, four heads. Launch and host latency are all there is.
        _case(name="forward_s128_h4_d64_fp16", heads=4, heads_k=4, head_dim=64, dtype="fp16"),
        # Decoding for one user: one query token against a filled 8k cache, grouped heads.
        _case(name="decode_b1_k8192", heads=32, heads_k=8, seqlen_q=1, seqlen_k=8192, causal=True, layout="cache"),
        # Decoding for a batch of users, an odd cache length.
        _case(name="decode_b32_k4093_fp16", batch=32, heads=32, heads_k=8, seqlen_q=1, seqlen_k=4093, causal=True,
              dtype="fp16", layout="cache"),
        # A chunk of a long prompt against what the cache already holds: ragged on both sides, bottom-right mask.
        _case(name="chunk_q1000_k9001", heads=32, heads_k=8, seqlen_q=1000, seqlen_k=9001, causal=True, layout="cache"),
        # The benchmark's forward: a batch of medium prompts.
        _case(name="prefill_b16_s2048", batch=16, seqlen_q=2048, seqlen_k=2048, causal=True),
        # Prefill of a sliding-window model.
        _case(name="prefill_window_b2_s8192", batch=2, heads=32, heads_k=8, seqlen_q=8192, seqlen_k=8192, causal=True,
              window=1023),
        # A small training step of a small model; results that have to be the same bits every time.
        _case(name="train_deterministic_b2_s777", kind="train", batch=2, heads=16, heads_k=4, seqlen_q=777, seqlen_k=777,
              causal=True, deterministic=True),
        # Training an encoder: short sequences just under a tile multiple, no mask, q, k and v are views of one projection.
        _case(name="train_encoder_b32_s509_d64_fp16", kind="train", batch=32, heads=12, heads_k=12, seqlen_q=509, seqlen_k=509,
              head_dim=64, dtype="fp16", layout="fused"),
        # The benchmark's training step.
        _case(name="train_b16_s2048", kind="train", batch=16, seqlen_q=2048, seqlen_k=2048, causal=True),
        # Training with soft-capped scores and grouped heads.
        _case(name="train_softcap_b4_s2048", kind="train", batch=4, heads=16, heads_k=4, seqlen_q=2048, seqlen_k=2048,
              causal=True, softcap=30.0),
        # Training with the widest head dim.
        _case(name="train_b4_s2048_d256", kind="train", batch=4, heads=16, heads_k=8, seqlen_q=2048, seqlen_k=2048,
              head_dim=256, causal=True),
        # Long-context training: the largest case.
        _case(name="train_b1_s16384", kind="train", heads=32, heads_k=32, seqlen_q=16384, seqlen_k=16384, causal=True),
    ]


def _log_int(rng, lo, hi):
    """An integer whose logarithm is spread evenly over [lo, hi]; odd as often as even."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.choice(("decode", "chunk", "prefill", "prefill", "train", "train", "train"))
    head_dim = rng.choice((64, 64, 96, 128, 128, 128, 128, 192, 256))
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    heads_k, group = rng.choice(((2, 1), (2, 4), (4, 1), (4, 4), (8, 1), (8, 2), (8, 4), (8, 8), (12, 1), (16, 1), (32, 1)))
    heads = heads_k * group
    case = _case(heads=heads, heads_k=heads_k, head_dim=head_dim, dtype=dtype)
    if what == "decode":
        # the cache of one layer: at most 2 GiB of K and V
        sk = _log_int(rng, 256, 32768)
        most = max(1, min(64, (1 << 31) // (sk * heads_k * head_dim * 4)))
        case.update(batch=_log_int(rng, 1, most), seqlen_q=rng.choice((1, 1, 1, 2, 4)), seqlen_k=sk, causal=True, layout="cache")
        return case
    if what == "chunk":
        sk = _log_int(rng, 1024, 16384)
        case.update(batch=rng.choice((1, 1, 2, 4)), seqlen_q=_log_int(rng, 64, min(2048, sk)), seqlen_k=sk, causal=True,
                    layout="cache")
        return case
    # at most a fifth of the operations of the largest listed case, without a mask
    per_pair = (14 if what == "train" else 4) * heads * head_dim
    s = _log_int(rng, 128, min(16384, math.isqrt(int(1.5e12 / per_pair))))
    causal = rng.random() < 0.75
    case.update(kind="train" if what == "train" else "forward", seqlen_q=s, seqlen_k=s, causal=causal,
                batch=_log_int(rng, 1, int(max(1, min(32, 1.5e12 // (per_pair * s * s))))))
    option = rng.choice(("none", "none", "none", "window", "softcap", "alibi", "deterministic", "fused"))
    if option == "window" and causal:
        case["window"] = rng.choice((127, 256, 1023, 4095))
    elif option == "softcap":
        case["softcap"] = rng.choice((15.0, 30.0, 50.0))
    elif option == "alibi":
        case["alibi"] = True
    elif option == "deterministic" and what == "train":
        case["deterministic"] = True
    elif option == "fused" and case["heads"] == case["heads_k"]:
        case["layout"] = "fused"
    return case


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = _DTYPES[case["dtype"]]
    b, sq, sk, h, hk, d = (case[n] for n in ("batch", "seqlen_q", "seqlen_k", "heads", "heads_k", "head_dim"))

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)

    if case["layout"] == "fused":
        q, k, v = normal(b, sq, 3, h, d).unbind(2)
    elif case["layout"] == "cache":
        room = (sk // 256 + 2) * 256  # the cache is allocated ahead of what it holds
        q, k, v = normal(b, sq, h, d), normal(b, room, hk, d)[:, :sk], normal(b, room, hk, d)[:, :sk]
    else:
        q, k, v = normal(b, sq, h, d), normal(b, sk, hk, d), normal(b, sk, hk, d)
    state = {"q": q, "k": k, "v": v, "kind": case["kind"], "alibi_slopes": None, "causal": case["causal"],
             "window": (case["window"], 0 if case["causal"] and case["window"] >= 0 else -1), "softcap": case["softcap"],
             "deterministic": case["deterministic"]}
    if case["alibi"]:
        state["alibi_slopes"] = torch.tensor([2.0 ** (-8.0 * (i + 1) / h) for i in range(h)], dtype=torch.float32, device="cuda")
    if case["kind"] == "train":
        for name in ("q", "k", "v"):
            state[name] = state[name].detach().requires_grad_(True)
        state["dout"] = normal(b, sq, h, d)
    return state


def run(state):
    q, k, v = state["q"], state["k"], state["v"]
    if state["kind"] == "forward":
        out, lse, _, _ = fa2.fwd(q, k, v, alibi_slopes=state["alibi_slopes"], is_causal=state["causal"],
                                 window_size_left=state["window"][0], window_size_right=state["window"][1],
                                 softcap=state["softcap"])
        return out, lse
    out = fa2.flash_attn_func(q, k, v, causal=state["causal"], window_size=state["window"], softcap=state["softcap"],
                              alibi_slopes=state["alibi_slopes"], deterministic=state["deterministic"])
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["dout"])
    return out.detach(), dq, dk, dv


def _pairs(case):
    """(query, key) pairs of one head that the mask leaves."""
    sq, sk, left = case["seqlen_q"], case["seqlen_k"], case["window"]
    if not case["causal"]:
        return sq * sk
    total = 0
    for i in range(sq):
        last = i + sk - sq
        total += max(0, last + 1 - (max(0, last - left) if left >= 0 else 0))
    return total


def work(case):
    b, sq, sk, h, hk, d = (case[n] for n in ("batch", "seqlen_q", "seqlen_k", "heads", "heads_k", "head_dim"))
    train = case["kind"] == "train"
    q_bytes, kv_bytes = 2 * b * sq * h * d, 2 * b * sk * hk * d
    # forward: read q, k, v, write the output and the LSE; training also reads dout and writes dq, dk and dv
    moved = 2 * q_bytes + 2 * kv_bytes + (2 * q_bytes + 2 * kv_bytes if train else 4 * b * h * sq)
    # two products forward, five backward
    return {"bytes": moved, "flops": (14 if train else 4) * b * h * _pairs(case) * d}


def tolerance(case):
    # Probabilities and score gradients are rounded to the input type on their way into the second product, and the
    # results are rounded to it: a few of the type's roundings (2^-9 for bf16, 2^-12 for fp16) in the 2-norm. The
    # hardware's tanh, which a soft cap multiplies by the cap, is good to 2^-11 only.
    if case["dtype"] == "bf16" or case["softcap"]:
        return {"rel": 1e-2}
    return {"rel": 2e-3}
