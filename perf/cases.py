"""The attention work a user of this package has it do, as cases that can be timed and compared.

Four entry points: ``F.scaled_dot_product_attention`` on the `mojo` device with PyTorch's autograd
behind it (training), the same call without gradients (prefill and decode), the aten operator that
also returns the logsumexp, and the two forwards on plain CUDA tensors in ``raw`` that take the
bottom-right causal alignment (new queries against a longer key/value cache).

A case: ``kind``; ``B, Hq, Hkv, Sq, Sk, D``; ``dtype``; ``mask`` ("none", "causal": torch's rule, the
diagonal starts top-left; "suffix": it ends bottom-right); ``fused`` (q, k, v are views of one
(B, S, 3*H*D) projection, as a transformer block makes them; else each is (B, H, S, D) contiguous);
``dropout``; ``std`` (spread of q, k and v).
"""

from __future__ import annotations

import torch
import torch.nn.functional as F

import torch_mojo_backend_b200 as tmb
from torch_mojo_backend_b200 import _lib, raw

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(kind, B, Hq, Hkv, Sq, Sk, D, dtype, mask, *, fused=False, dropout=0.0, std=0.5):
    return {"kind": kind, "B": B, "Hq": Hq, "Hkv": Hkv, "Sq": Sq, "Sk": Sk, "D": D, "dtype": dtype,
            "mask": mask, "fused": fused, "dropout": dropout, "std": std}


def listed():
    return [
        # training attention of a GPT-2-small block: q, k and v are views of the block's fused projection
        {"name": "gpt2-train-bf16", **_case("train", 8, 12, 12, 1024, 1024, 64, "bf16", "causal", fused=True, std=1.0)},
        # the same block kept in fp32, as a script without autocast runs it, at a smaller batch
        {"name": "gpt2-train-fp32", **_case("train", 4, 12, 12, 1024, 1024, 64, "fp32", "causal", fused=True, std=1.0)},
        # Llama-style grouped-query training step at a 4k context
        {"name": "llama-train-bf16", **_case("train", 4, 32, 8, 4096, 4096, 128, "bf16", "causal")},
        # one large unmasked fp16 batch, forward and backward: as much as one GPU of a data-parallel job is given
        {"name": "batch-train-fp16", **_case("train", 64, 16, 16, 2048, 2048, 128, "fp16", "none", std=0.577)},
        # variable-length fine-tuning: a length that fits no tile, dropout, grouped heads
        {"name": "ragged-dropout-bf16", **_case("train", 5, 16, 4, 777, 777, 128, "bf16", "causal", dropout=0.1)},
        # cross-attention of an encoder-decoder: few keys, both lengths ragged
        {"name": "cross-train-fp16", **_case("train", 16, 8, 8, 1000, 77, 64, "fp16", "none")},
        # long-context prefill of one prompt
        {"name": "long-prefill-bf16", **_case("forward", 1, 32, 32, 32768, 32768, 128, "bf16", "causal", std=1.0)},
        # a small exact-fp32 evaluation that wants the logsumexp too: a call of this size is latency
        {"name": "small-eval-fp32", **_case("forward_lse", 2, 4, 4, 256, 256, 64, "fp32", "causal", std=1.0)},
        # chunked prefill: the next 512 tokens of a prompt against what is already in the cache
        {"name": "chunk-prefill-bf16", **_case("chunk", 1, 32, 8, 512, 16896, 128, "bf16", "suffix")},
        # one decoding step of a batch with long caches
        {"name": "decode-long-bf16", **_case("forward", 8, 32, 8, 1, 32768, 128, "bf16", "none")},
        # one decoding step of an ordinary chat: caches of a thousand tokens
        {"name": "decode-chat-fp16", **_case("forward", 4, 32, 8, 1, 1000, 128, "fp16", "none")},
        # four drafted tokens per sequence verified at once against the cache
        {"name": "verify-bf16", **_case("verify", 16, 32, 8, 4, 16384, 128, "bf16", "suffix")},
    ]


_MOST_FLOPS = 7.6e12    # no more than the largest listed case
_MOST_VALUES = 5.5e8    # elements of q, k and v together


def _length(rng, lo, hi):
    """Spread over the logarithm of the range; a round number as often as not."""
    n = int(round(lo * (hi / lo) ** rng.random()))
    if rng.random() < 0.5:
        n = max(lo, n // 64 * 64) if n >= 128 else n
    return max(1, n)


def _heads(rng):
    """(query heads, key/value heads)"""
    hkv = rng.choice([1, 2, 4, 6, 8, 12, 16])
    return hkv * rng.choice([1, 1, 2, 3, 4, 8]), hkv


def draw(rng):
    while True:
        kind = rng.choice(["train", "train", "train", "forward", "forward", "forward_lse", "chunk", "decode", "decode",
                           "verify"])
        hq, hkv = _heads(rng)
        d = rng.choice([64, 128])
        dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
        std = rng.choice([0.5, 0.577, 1.0])
        b = _length(rng, 1, 64)
        if kind == "train":
            sq = _length(rng, 64, 8192)
            mask = rng.choice(["causal", "causal", "none"])
            sk = sq if mask == "causal" or rng.random() < 0.7 else _length(rng, 16, 8192)
            c = _case(kind, b, hq, hkv, sq, sk, d, dtype, mask, fused=sq == sk and rng.random() < 0.5,
                      dropout=rng.choice([0.0, 0.0, 0.0, 0.1, 0.2]), std=std)
        elif kind in ("forward", "forward_lse"):
            s = _length(rng, 64, 32768)
            c = _case(kind, b, hq, hkv, s, s, d, dtype, rng.choice(["causal", "causal", "none"]), std=std)
        elif kind == "chunk":
            sq = _length(rng, 32, 2048)
            c = _case(kind, b, hq, hkv, sq, sq + _length(rng, 128, 32768), d, dtype, "suffix", std=std)
        elif kind == "decode":
            c = _case("forward", b, hq, hkv, 1, _length(rng, 64, 131072), d, dtype, "none", std=std)
        else:
            sq = rng.choice([2, 3, 4, 5])
            if hq // hkv * sq > _lib.SPLITKV_MAX_ROWS:
                continue
            c = _case(kind, b, hq, hkv, sq, _length(rng, 512, 131072), d, dtype, "suffix", std=std)
        values = b * d * (hq * c["Sq"] + 2 * hkv * c["Sk"])
        # fp32 runs on the fp32 units: a fraction of the 16-bit rate, so a fraction of the work
        most = _MOST_FLOPS / (100 if dtype == "fp32" else 1)
        if work(c)["flops"] <= most and values * (2 if dtype == "fp32" else 1) <= _MOST_VALUES:
            return c


def _randn(gen, shape, std, dtype):
    """Normal values of the given spread, rounded to the case's type."""
    t = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32 if dtype == torch.float32 else torch.float16)
    return t.mul_(std).to(dtype)


def _inputs(case, seed):
    """q, k, v as (B, H, S, D) views, and the upstream gradient of a training case."""
    B, Hq, Hkv, Sq, Sk, D = (case[n] for n in ("B", "Hq", "Hkv", "Sq", "Sk", "D"))
    dtype, std = _DTYPES[case["dtype"]], case["std"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["fused"]:
        proj = _randn(gen, (B, Sq, (Hq + 2 * Hkv) * D), std, dtype)
        q, k, v = (p.unflatten(2, (-1, D)).transpose(1, 2) for p in proj.split([Hq * D, Hkv * D, Hkv * D], dim=2))
    else:
        q = _randn(gen, (B, Hq, Sq, D), std, dtype)
        k, v = (_randn(gen, (B, Hkv, Sk, D), std, dtype) for _ in range(2))
    grad = None
    if case["kind"] == "train":
        # the gradient arrives in the layout the output is handed on in: (B, S, H, D) behind a fused projection
        grad = (_randn(gen, (B, Sq, Hq, D), 1.0, dtype).transpose(1, 2) if case["fused"]
                else _randn(gen, (B, Hq, Sq, D), 1.0, dtype))
    return q, k, v, grad


def prepare(case, seed):
    tmb.register_mojo_devices()
    q, k, v, grad = _inputs(case, seed)
    kind = case["kind"]
    state = {"kind": kind, "q": q, "k": k, "v": v, "causal": case["mask"] == "causal", "scale": case["D"] ** -0.5,
             "dropout": case["dropout"], "gqa": case["Hq"] != case["Hkv"]}
    if kind in ("chunk", "verify"):
        return state
    q, k, v = (tmb.from_cuda(t) for t in (q, k, v))
    if kind == "train":
        torch.mojo.manual_seed(seed)   # where the dropout masks of this state's passes start
        state["grad"] = tmb.from_cuda(grad)
        q, k, v = (t.requires_grad_() for t in (q, k, v))
    state.update(q=q, k=k, v=v)
    return state


def run(state):
    kind, q, k, v = state["kind"], state["q"], state["k"], state["v"]
    if kind == "train":
        out = F.scaled_dot_product_attention(q, k, v, dropout_p=state["dropout"], is_causal=state["causal"],
                                             enable_gqa=state["gqa"])
        dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["grad"])
        return {"out": tmb.to_cuda(out.detach()), "dq": tmb.to_cuda(dq), "dk": tmb.to_cuda(dk), "dv": tmb.to_cuda(dv)}
    if kind == "forward":
        with torch.no_grad():
            return {"out": tmb.to_cuda(F.scaled_dot_product_attention(q, k, v, is_causal=state["causal"],
                                                                      enable_gqa=state["gqa"]))}
    if kind == "forward_lse":
        with torch.no_grad():
            res = torch.ops.aten._scaled_dot_product_flash_attention(q, k, v, 0.0, state["causal"], scale=state["scale"])
        return {"out": tmb.to_cuda(res[0]), "lse": tmb.to_cuda(res[1])}
    forward = raw.flash_fwd if kind == "chunk" else raw.flash_fwd_splitkv
    out, lse = forward(q, k, v, causal=_lib.CAUSAL_BOTTOM_RIGHT)
    return {"out": out, "lse": lse}


_EXACT_SCORES = 1 << 28   # 64-bit scores held at a time


def exact(case, seed):
    """The same outputs in 64 bits, one key/value head at a time and as many query rows as fit."""
    if case["dropout"]:
        return None   # the mask is this package's own random stream
    B, Hq, Hkv, Sq, Sk, D = (case[n] for n in ("B", "Hq", "Hkv", "Sq", "Sk", "D"))
    if 8 * B * Hq * Sq * Sk * D > 1e14:
        return None   # too long in 64 bits
    q, k, v, grad = _inputs(case, seed)
    group, scale, kind = Hq // Hkv, D ** -0.5, case["kind"]
    f64 = {"dtype": torch.float64, "device": "cuda"}
    res = {"out": torch.empty((B, Hq, Sq, D), **f64)}
    if kind == "train":
        res.update(dq=torch.empty((B, Hq, Sq, D), **f64), dk=torch.zeros((B, Hkv, Sk, D), **f64),
                   dv=torch.zeros((B, Hkv, Sk, D), **f64))
    elif kind != "forward":
        res["lse"] = torch.empty((B, Hq, Sq), **f64)
    rows = max(1, _EXACT_SCORES // (group * Sk))
    col = torch.arange(Sk, device="cuda")
    for b in range(B):
        for h in range(Hkv):
            heads = slice(h * group, (h + 1) * group)
            k64, v64 = k[b, h].double(), v[b, h].double()
            for r0 in range(0, Sq, rows):
                r = slice(r0, min(Sq, r0 + rows))
                q64 = q[b, heads, r].double() * scale
                s = q64 @ k64.T
                if case["mask"] != "none":
                    last = torch.arange(r.start, r.stop, device="cuda") + (Sk - Sq if case["mask"] == "suffix" else 0)
                    s.masked_fill_(col > last[:, None], -torch.inf)
                lse = torch.logsumexp(s, dim=-1)
                p = s.sub_(lse[..., None]).exp_()
                o = p @ v64
                res["out"][b, heads, r] = o
                if kind == "train":
                    g = grad[b, heads, r].double()
                    res["dv"][b, h] += torch.einsum("gqk,gqd->kd", p, g)
                    ds = p.mul_((g @ v64.T).sub_((g * o).sum(-1, keepdim=True)))
                    res["dq"][b, heads, r] = ds @ k64 * scale
                    res["dk"][b, h] += torch.einsum("gqk,gqd->kd", ds, q64)
                elif kind != "forward":
                    res["lse"][b, heads, r] = lse
    return res


def _visible(case):
    """(query, key) pairs that take part, per head."""
    Sq, Sk = case["Sq"], case["Sk"]
    if case["mask"] == "none":
        return Sq * Sk
    if case["mask"] == "causal":
        n = min(Sq, Sk)
        return n * (n + 1) // 2 + (Sq - n) * Sk
    return Sq * (Sk - Sq) + Sq * (Sq + 1) // 2


def work(case):
    B, Hq, Hkv, Sq, Sk, D = (case[n] for n in ("B", "Hq", "Hkv", "Sq", "Sk", "D"))
    size = 4 if case["dtype"] == "fp32" else 2
    q, kv = B * Hq * Sq * D * size, 2 * B * Hkv * Sk * D * size
    forward = 4 * B * Hq * _visible(case) * D
    if case["kind"] == "train":
        # q, k, v, the upstream gradient in; the output, dq, dk, dv out
        return {"bytes": 4 * q + 2 * kv, "flops": 3.5 * forward}
    lse = 0 if case["kind"] == "forward" else 4 * B * Hq * Sq
    return {"bytes": 2 * q + kv + lse, "flops": forward}


def tolerance(case):
    # 16-bit types: the probabilities and their gradients are rounded to the type before they are
    # multiplied on, and every result is rounded to it.  Against the same attention in 64 bits (2-norms;
    # the worst of out, dq, dk, dv over the listed cases, lengths up to 1024): bf16 2.5e-3, fp16 3.0e-4,
    # fp32 8.0e-7, growing with the length in fp32 (sums of up to 100 times as many terms are drawn).
    return {"rel": {"bf16": 1e-2, "fp16": 1.2e-3, "fp32": 5e-6}[case["dtype"]]}
