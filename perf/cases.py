"""The work whose speed this framework is judged by: attention prefill, training steps, decoding over dense, block-sparse
and latent (MLA) caches, and chunked linear attention, all through the public entry points, at sizes from the
repository's own benchmark and tests and at odd ones in between.

Every case is a dict of plain values; ``draw`` gives further cases of the same ranges.  Inputs are drawn on the GPU from
the seed with the distributions of ``oracle/inputs.py`` (N(0, 1) activations, RetNet / gated / Mamba2 decays)."""

from __future__ import annotations

import math

import torch

import metaattention_b200  # noqa: F401  (makes attn_engine, core and examples_b200 importable)
from attn_engine import AttentionEngine
from attn_engine.mla import flash_mla_with_kvcache, get_mla_metadata
from core import CustomIO, meta_tensor
from examples_b200 import programs

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


# ---------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------

def _attention(kind, dtype, B, H, Hkv, S, D, Dv, mask, window=0):
    return {"kind": kind, "dtype": dtype, "B": B, "H": H, "Hkv": Hkv, "S": S, "D": D, "Dv": Dv, "mask": mask, "window": window}


def _decode(dtype, B, H, Hkv, S, D, q_len=1):
    return {"kind": "decode", "dtype": dtype, "B": B, "H": H, "Hkv": Hkv, "S": S, "D": D, "q_len": q_len}


def _linear(kind, dtype, program, B, H, S, Dk, Dv):
    return {"kind": kind, "dtype": dtype, "program": program, "B": B, "H": H, "S": S, "Dk": Dk, "Dv": Dv}


def listed():
    return [
        # A short prompt on a small model with grouped KV heads: microseconds of work, all latency and launches.
        dict(_attention("prefill", "fp16", 1, 16, 4, 333, 64, 64, "causal"), name="prefill_short"),
        # The configuration the benchmark's headline is quoted on: a large causal prefill.
        dict(_attention("prefill", "bf16", 8, 32, 32, 4096, 128, 128, "causal"), name="prefill_large"),
        # Prefill of a latent-attention model, whose queries and keys are wider (128 + 64 rope) than its values.
        dict(_attention("prefill", "bf16", 2, 16, 16, 3000, 192, 128, "causal"), name="prefill_192_128"),
        # Sigmoid attention (a lowered score_mod with a bias, no online function), bidirectional: vision-style encoders.
        dict(_attention("prefill_sigmoid", "bf16", 2, 32, 32, 4096, 128, 128, "none"), name="prefill_sigmoid"),
        # Training step (forward and all gradients) of a causal language model.
        dict(_attention("train", "bf16", 4, 32, 32, 4096, 128, 128, "causal"), name="train_causal"),
        # Training step of a small model with a sliding window and grouped heads on a ragged length.
        dict(_attention("train", "fp16", 2, 16, 4, 1111, 64, 64, "window", 256), name="train_small_window"),
        # One token against one long context, every head with its own cache: latency of long-context generation.
        dict(_decode("bf16", 1, 32, 32, 32768, 128), name="decode_mha_long"),
        # Batched generation with grouped KV heads over caches of different lengths of which a part of the blocks is kept.
        {"name": "decode_gqa_sparse", "kind": "decode_sparse", "dtype": "bf16", "B": 8, "H": 32, "Hkv": 8, "S": 8192, "D": 128,
         "block": 32, "kept": 0.3},
        # Batched MLA generation over a paged latent cache with ragged lengths, one layer's call with the step's schedule.
        {"name": "mla_paged", "kind": "mla", "dtype": "bf16", "B": 64, "H": 128, "S": 8192, "paged": True},
        # RetNet retention at the benchmark's configuration.
        dict(_linear("linear", "bf16", "retnet", 8, 8, 4096, 256, 512), name="retention_large"),
        # Mamba2 state-space mixing of one sequence: 80 value heads of 64 columns on one q / k group.
        dict(_linear("linear", "bf16", "mamba2", 1, 80, 2048, 128, 64), name="mamba2"),
        # Training step of gated retention: gradients of q, k, v and of the learned gates.
        dict(_linear("linear_train", "bf16", "gla", 2, 8, 2000, 128, 256), name="train_gated_retention"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_once(rng):
    kind = rng.choice(["prefill", "prefill", "prefill_sigmoid", "train", "train", "train_sigmoid", "decode", "decode", "decode_sparse",
                       "mla", "linear", "linear", "linear_train"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind in ("prefill", "prefill_sigmoid", "train", "train_sigmoid"):
        train = kind.startswith("train")
        H = rng.choice([8, 16, 32])
        Hkv = rng.choice([H, H, H // 4])
        S = _log_int(rng, 128, 4096)
        D, Dv = rng.choice([(64, 64), (128, 128), (128, 128)] + ([] if kind != "prefill" else [(192, 128), (256, 256)]))
        mask = rng.choice(["causal", "none"] if kind.endswith("sigmoid") else ["causal", "causal", "none", "window", "document"])
        window = _log_int(rng, 64, max(128, S // 2)) if mask in ("window", "document") else 0
        return _attention(kind, dtype, rng.randint(1, 4 if train else 8), H, Hkv, S, D, Dv, mask, window)
    if kind == "decode":
        Hkv = rng.choice([32, 8, 8, 4])
        return _decode(dtype, _log_int(rng, 1, 32), 32, Hkv, _log_int(rng, 512, 32768), rng.choice([64, 128, 128]), rng.choice([1, 1, 1, 4]))
    if kind == "decode_sparse":
        return {"kind": kind, "dtype": dtype, "B": _log_int(rng, 1, 32), "H": 32, "Hkv": rng.choice([8, 4]), "S": 64 * _log_int(rng, 16, 256),
                "D": 128, "block": rng.choice([32, 64]), "kept": round(rng.uniform(0.1, 1.0), 2)}
    if kind == "mla":
        return {"kind": kind, "dtype": dtype, "B": _log_int(rng, 1, 128), "H": rng.choice([64, 128, 128]), "S": 64 * _log_int(rng, 8, 128),
                "paged": rng.choice([True, False])}
    program = rng.choice(["retnet", "gla"] if kind == "linear_train" else ["retnet", "gla", "mamba2"])
    S = _log_int(rng, 256, 4096)
    if program == "mamba2":
        return _linear(kind, dtype, program, rng.randint(1, 2), rng.choice([24, 64, 80]), S, rng.choice([64, 128]), 64)
    Dk, Dv = rng.choice([(64, 128), (128, 128), (128, 256), (256, 256), (256, 512)])
    return _linear(kind, dtype, program, rng.randint(1, 8), rng.choice([4, 8, 16]), S, Dk, Dv)


def draw(rng):
    top = [work(c) for c in listed()]
    most_flops, most_bytes = max(w["flops"] for w in top), max(w["bytes"] for w in top)
    while True:
        case = _draw_once(rng)
        w = work(case)
        # gradients of linear attention cost more time for their operations than any other kind
        share = 0.25 if case["kind"] == "linear_train" else 1.0
        if w["flops"] <= share * most_flops and w["bytes"] <= share * most_bytes:
            return case


# ---------------------------------------------------------------------------------------------------------------
# what a user's program has in hand before the call
# ---------------------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(gen, *shape, dtype, scale=1.0):
    t = torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)
    return t if scale == 1.0 else t * scale


def _mask_mod(mask, window):
    if mask == "causal":
        return programs.causal
    if mask == "window":
        return lambda b, h, q_idx, kv_idx: (q_idx >= kv_idx) & (q_idx - kv_idx < window)
    if mask == "document":   # packed documents of `window` tokens, causal inside each
        return lambda b, h, q_idx, kv_idx: (q_idx // window == kv_idx // window) & (q_idx >= kv_idx)
    return None


def _metas(B, H, Hkv, Sq, Skv, D, Dv, dtype):
    return (meta_tensor(B, H, Sq, D, dtype=dtype), meta_tensor(B, Hkv, Skv, D, dtype=dtype), meta_tensor(B, Hkv, Skv, Dv, dtype=dtype))


def _softmax_engine(metas, scale, mask_mod=None, **kwargs):
    def score_mod(score, custom, b, h, q_idx, kv_idx):
        return score * scale
    return AttentionEngine(metas, CustomIO({}), score_mod=score_mod, mask_mod=mask_mod, online_func=programs.NaturalSoftmax(), **kwargs)


def _sigmoid_engine(metas, scale, mask_mod=None):
    def score_mod(score, custom, b, h, q_idx, kv_idx):
        x = score * scale + custom.input_tensors["softmax_bias"]
        return ((x * 0.5).tanh() + 1) * 0.5
    return AttentionEngine(metas, CustomIO({"softmax_bias": (1,)}), score_mod=score_mod, mask_mod=mask_mod, online_func=None)


def _prepare_attention(c, gen, dtype):
    B, H, Hkv, S, D, Dv = c["B"], c["H"], c["Hkv"], c["S"], c["D"], c["Dv"]
    metas, mask_mod = _metas(B, H, Hkv, S, S, D, Dv, dtype), _mask_mod(c["mask"], c["window"])
    st = {"q": _randn(gen, B, S, H, D, dtype=dtype), "k": _randn(gen, B, S, Hkv, D, dtype=dtype), "v": _randn(gen, B, S, Hkv, Dv, dtype=dtype),
          "custom": ()}
    if c["kind"].endswith("sigmoid"):
        st["engine"] = _sigmoid_engine(metas, D ** -0.5, mask_mod)
        st["custom"] = (torch.tensor([-math.log(S)], device="cuda"),)
    else:
        st["engine"] = _softmax_engine(metas, D ** -0.5, mask_mod)
    if c["kind"].startswith("train"):
        st["d_o"] = _randn(gen, B, S, H, Dv, dtype=dtype)
        for name in ("q", "k", "v"):
            st[name].requires_grad_()
    return st


def _prepare_decode(c, gen, dtype):
    B, H, Hkv, S, D, q_len = c["B"], c["H"], c["Hkv"], c["S"], c["D"], c["q_len"]
    return {"q": _randn(gen, B, q_len, H, D, dtype=dtype), "k": _randn(gen, B, S, Hkv, D, dtype=dtype),
            "v": _randn(gen, B, S, Hkv, D, dtype=dtype), "engine": _softmax_engine(_metas(B, H, Hkv, q_len, S, D, D, dtype), D ** -0.5)}


def _prepare_decode_sparse(c, gen, dtype):
    B, H, Hkv, S, D, block = c["B"], c["H"], c["Hkv"], c["S"], c["D"], c["block"]
    engine = _softmax_engine(_metas(B, H, Hkv, 1, S, D, D, dtype), D ** -0.5, extern_block_mask=True, use_varlen=True, infer_mask_block_N=block)
    lens = torch.randint(S // 4, S + 1, (B,), generator=gen, device="cuda", dtype=torch.int32)
    blocks = S // block
    keep = torch.rand(B, Hkv, blocks, generator=gen, device="cuda") < c["kept"]
    keep[..., 0] = True   # the first block and the one with the newest token are always kept
    keep |= (torch.arange(blocks, device="cuda") == ((lens - 1) // block)[:, None])[:, None]
    return {"q": _randn(gen, B, 1, H, D, dtype=dtype), "k": _randn(gen, B, S, Hkv, D, dtype=dtype),
            "v": _randn(gen, B, S, Hkv, D, dtype=dtype), "engine": engine, "block_mask": keep, "lens": lens}


def _prepare_mla(c, gen, dtype):
    B, H, S, D, Dv, page = c["B"], c["H"], c["S"], 576, 512, 64
    st = {"q": _randn(gen, B, 1, H, D, dtype=dtype)}
    if c["paged"]:
        per_seq = S // page
        st["cache"] = _randn(gen, B * per_seq, page, 1, D, dtype=dtype)
        st["lens"] = torch.randint(S // 8, S + 1, (B,), generator=gen, device="cuda", dtype=torch.int32)
        st["table"] = torch.randperm(B * per_seq, generator=gen, device="cuda").view(B, per_seq).to(torch.int32)
        # made once per decoding step, used by every layer
        st["metadata"], st["num_splits"] = get_mla_metadata(st["lens"], H)
    else:
        st["kv"], st["k_pe"] = _randn(gen, B, S, 1, Dv, dtype=dtype), _randn(gen, B, S, 1, D - Dv, dtype=dtype)
        st["q_nope"], st["q_pe"] = st["q"][..., :Dv].contiguous(), st["q"][..., Dv:].contiguous()
        st["engine"] = programs.mla_engine(B, H, S, D, Dv, dtype=dtype)
    return st


def _prepare_linear(c, gen, dtype):
    B, H, S, Dk, Dv, program = c["B"], c["H"], c["S"], c["Dk"], c["Dv"], c["program"]
    Hq = 1 if program == "mamba2" else H
    k_scale = {"retnet": Dk ** -0.5, "gla": 1.0, "mamba2": 0.5}[program]
    st = {"q": _randn(gen, B, Hq, S, Dk, dtype=dtype), "k": _randn(gen, B, Hq, S, Dk, dtype=dtype, scale=k_scale),
          "v": _randn(gen, B, H, S, Dv, dtype=dtype), "custom": ()}
    if program == "retnet":
        gamma = 1.0 - torch.exp2(-5.0 - torch.arange(H, dtype=torch.float32, device="cuda") % 8)
        st["decay"] = gamma[None, :, None].expand(B, H, S).contiguous()
        st["engine"] = programs.retnet_engine(B, H, S, Dk, Dv, dtype=dtype)
    elif program == "gla":
        st["decay"] = torch.nn.functional.logsigmoid(torch.randn(B, H, S, generator=gen, device="cuda")).clamp_min(-5.0)
        st["engine"] = programs.gla_engine(B, H, S, Dk, Dv, dtype=dtype)
    else:
        A = 1.5 * torch.rand(1, H, generator=gen, device="cuda") - 4.0
        dt0 = torch.exp(torch.rand(H, generator=gen, device="cuda") * math.log(100.0) + math.log(0.001)).clamp(min=1e-4)
        bias = dt0 + torch.log(-torch.expm1(-dt0))
        st["decay"] = torch.nn.functional.softplus(0.7 * torch.rand(B, H, S, generator=gen, device="cuda") + bias.view(1, H, 1))
        st["custom"] = (A, st["decay"])
        st["engine"] = programs.mamba2_engine(B, 1, S, Dk, Dv, HV=H, dtype=dtype)
    if c["kind"] == "linear_train":
        st["d_o"] = _randn(gen, B, H, S, Dv, dtype=dtype)
        for name in ("q", "k", "v") + (("decay",) if program == "gla" else ()):   # RetNet's decays are constants
            st[name].requires_grad_()
    return st


def prepare(case, seed):
    gen, dtype = _gen(seed), DTYPES[case["dtype"]]
    kind = case["kind"]
    if kind == "decode":
        st = _prepare_decode(case, gen, dtype)
    elif kind == "decode_sparse":
        st = _prepare_decode_sparse(case, gen, dtype)
    elif kind == "mla":
        st = _prepare_mla(case, gen, dtype)
    elif kind in ("linear", "linear_train"):
        st = _prepare_linear(case, gen, dtype)
    else:
        st = _prepare_attention(case, gen, dtype)
    st["case"] = case
    return st


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------

def run(st):
    kind = st["case"]["kind"]
    if kind in ("prefill", "prefill_sigmoid"):
        o = st["engine"](st["q"], st["k"], st["v"], *st["custom"])
        return [o, *st["engine"].last_final_rowscales.values()]
    if kind in ("train", "train_sigmoid"):
        o = st["engine"](st["q"], st["k"], st["v"], *st["custom"])
        return [o.detach(), *torch.autograd.grad(o, (st["q"], st["k"], st["v"]), st["d_o"])]
    if kind == "decode":
        o = st["engine"](st["q"], st["k"], st["v"])
        return [o, st["engine"].last_final_rowscales["lse"]]
    if kind == "decode_sparse":
        o = st["engine"](st["q"], st["k"], st["v"], block_mask=st["block_mask"], cache_seqlens=st["lens"])
        return [o, st["engine"].last_final_rowscales["lse"]]
    if kind == "mla":
        if st["case"]["paged"]:
            return list(flash_mla_with_kvcache(st["q"], st["cache"], st["table"], st["lens"], 512, st["metadata"], st["num_splits"]))
        o = st["engine"](st["q_nope"], st["q_pe"], st["kv"], st["k_pe"])
        return [o, st["engine"].last_final_rowscales["lse"]]
    o = st["engine"](st["q"], st["k"], st["v"], st["decay"], *st["custom"])
    if kind == "linear":
        return [o]
    leaves = [st["q"], st["k"], st["v"]] + ([st["decay"]] if st["decay"].requires_grad else [])
    return [o.detach(), *torch.autograd.grad(o, leaves, st["d_o"])]


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far correct results may lie apart
# ---------------------------------------------------------------------------------------------------------------

def _kept_pairs(mask, S, window):
    """(query, key) pairs a mask keeps."""
    if mask == "causal":
        return S * (S + 1) / 2
    if mask == "window":
        w = min(window, S)
        return w * (w + 1) / 2 + (S - w) * w
    if mask == "document":
        whole, rest = divmod(S, window)
        return whole * window * (window + 1) / 2 + rest * (rest + 1) / 2
    return float(S) * S


def work(case):
    c, kind = case, case["kind"]
    if kind in ("prefill", "prefill_sigmoid", "train", "train_sigmoid"):
        B, H, Hkv, S, D, Dv = c["B"], c["H"], c["Hkv"], c["S"], c["D"], c["Dv"]
        tensors = B * S * (H * (D + Dv) + Hkv * (D + Dv)) * 2.0      # q, k, v in, o out
        flops = 2.0 * B * H * _kept_pairs(c["mask"], S, c["window"]) * (D + Dv)
        if kind.startswith("train"):   # + dO in, dq, dk, dv out; five products of the backward on top of the forward's two
            return {"bytes": 2 * tensors, "flops": 3.5 * flops}
        return {"bytes": tensors + 4.0 * B * H * S, "flops": flops}
    if kind in ("decode", "decode_sparse"):
        B, H, Hkv, S, D, q_len = c["B"], c["H"], c["Hkv"], c["S"], c["D"], c.get("q_len", 1)
        share = 1.0 if kind == "decode" else 0.625 * c["kept"]       # lengths are uniform in [S/4, S]
        return {"bytes": 4.0 * B * Hkv * S * D * share + 4.0 * B * q_len * H * D, "flops": 4.0 * B * H * q_len * S * D * share}
    if kind == "mla":
        B, H, S = c["B"], c["H"], c["S"]
        tokens = B * S * (0.5625 if c["paged"] else 1.0)             # lengths are uniform in [S/8, S]
        return {"bytes": 2.0 * (tokens * 576 + B * H * (576 + 512)), "flops": 2.0 * H * tokens * (576 + 512)}
    B, H, S, Dk, Dv = c["B"], c["H"], c["S"], c["Dk"], c["Dv"]
    Hq = 1 if c["program"] == "mamba2" else H
    tensors = 2.0 * B * S * (2 * Hq * Dk + 2 * H * Dv) + 4.0 * B * H * S
    flops = B * H * S * (2.0 * 64 * (Dk + Dv) + 4.0 * Dk * Dv)       # chunks of 64 tokens
    # gradients: five products where the forward has two
    return {"bytes": 2 * tensors, "flops": 3.5 * flops} if kind == "linear_train" else {"bytes": tensors, "flops": flops}


# Largest relative error (2-norm) against the same path in 64 bits over all kinds and outputs: 2.9e-3 in bf16, 3.6e-4 in
# fp16; the gates' gradient of linear attention, a running sum of differences, 5.1e-3 and 6.9e-4.  Four times that.
def tolerance(case):
    gates = case["kind"] == "linear_train" and case["program"] == "gla"
    if case["dtype"] == "bf16":
        return {"rel": 2e-2 if gates else 1.2e-2}
    return {"rel": 2.8e-3 if gates else 1.5e-3}
