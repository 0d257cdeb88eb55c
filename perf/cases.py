"""Performance cases of the attention operator: what a user of the package has it do, through its public entry points.

A case is a dict of plain values:

  entry    "op":     twopass_attention / twopass_attention_train on q, k, v [B, H, N, D]
           "packed": twopass_attention_qkvpacked on a projection output [B, N, 3, H, D], the call of the ViT and Swin hooks
  train    forward + backward (out, every gradient, the bias gradient where there is a bias) or the forward alone
  b h n d  batch (images, or images x windows), heads, tokens, head dim
  dtype    float16, bfloat16, float32
  causal   lower-triangular mask
  bias     "none", or "heads": one additive fp32 bias per head, shared by the batch ([1, H, N, N])
"""
from __future__ import annotations

import math

import torch

from elsa_b200 import twopass_attention, twopass_attention_train
from elsa_b200.attention_bwd import twopass_attention_qkvpacked

WINDOW_TOKENS = 64          # a sequence of at most this many tokens with a bias is an attention window
ROWS_MAX = 131072           # batch x heads x tokens of an ordinary problem (the long fp32 one has more)
SCORES_MAX = 1 << 27        # elements of a drawn bias: heads x tokens x tokens


def _case(entry, train, b, h, n, d, dtype, causal=False, bias="none", name=None):
    c = {"entry": entry, "train": train, "b": b, "h": h, "n": n, "d": d, "dtype": dtype, "causal": causal, "bias": bias}
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # one 224 x 224 image through ViT-Tiny, inference: the smallest call, latency and launches count
        _case("packed", False, 1, 3, 197, 64, "float16", name="vit224_b1_infer"),
        # ViT-Tiny training at 224 x 224, 64 images: many short ragged sequences
        _case("packed", True, 64, 3, 197, 64, "float16", name="vit224_b64_train"),
        # ViT-Tiny training at 1024 x 1024 (64 x 64 patches and the class token): long, ragged by one token
        _case("packed", True, 8, 3, 4097, 64, "float16", name="vit1024_b8_train"),
        # Swin-T training, stage 1: 8 images x 64 windows of 7 x 7 tokens with the relative-position bias and its gradient
        _case("packed", True, 512, 3, 49, 32, "float16", bias="heads", name="swin_s1_train"),
        # Swin-T training, stage 4: one window per image, 24 heads; so little work that the host path counts
        _case("packed", True, 8, 24, 49, 32, "float16", bias="heads", name="swin_s4_train"),
        # long-context training step of one layer, fp16: the benchmark's headline workload
        _case("op", True, 1, 8, 16384, 64, "float16", name="long_fp16_train"),
        # causal (decoder) training step, bf16
        _case("op", True, 1, 8, 16384, 64, "bfloat16", causal=True, name="causal_bf16_train"),
        # fp32 inference at a thousand tokens
        _case("op", False, 1, 8, 1024, 64, "float32", name="fp32_1k_infer"),
        # fp32 training at a few thousand tokens
        _case("op", True, 1, 8, 4096, 64, "float32", name="fp32_4k_train"),
        # very long fp32 training step on one GPU: the largest case
        _case("op", True, 1, 8, 65536, 64, "float32", name="fp32_64k_train"),
        # head dim 128, the wide-head kernels
        _case("op", True, 1, 8, 8192, 128, "float16", name="d128_8k_train"),
        # a dense per-head bias on a long sequence, with its gradient
        _case("op", True, 1, 8, 4096, 64, "float16", bias="heads", name="bias_4k_train"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _batch(rng, h, n, most=64):
    return _log_int(rng, 1, max(1, min(most, ROWS_MAX // (h * n))))


def draw(rng):
    """One more case of the same ranges: a ViT layer, a set of attention windows, a plain attention call, or a biased one."""
    kind = rng.choice(("vit", "windows", "op", "op", "op", "bias"))
    train = rng.random() < 0.7
    half = rng.choice(("float16", "bfloat16"))
    if kind == "vit":           # side x side patches and, as a rule, a class token: 224 to 1024 pixels at patch size 16
        side = _log_int(rng, 14, 64)
        n = side * side + rng.choice((0, 1, 1, 1))
        h = rng.choice((3, 6, 12))
        return _case("packed", train, _batch(rng, h, n), h, n, 64, half)
    if kind == "windows":       # 7 x 7 or 8 x 8 windows: (images x windows) x heads as in the four Swin stages
        h = rng.choice((3, 6, 12, 24))
        n = rng.choice((49, 49, 64))
        return _case("packed", train, 8 * _log_int(rng, 1, 192 // h), h, n, 32, half, bias="heads")
    if kind == "op":
        dtype = rng.choice(("float16", "bfloat16", "float32"))
        d = rng.choice((32, 64, 64)) if dtype == "float32" else rng.choice((32, 64, 64, 96, 128))
        h = rng.choice((4, 8, 8, 16))
        longest = 32768 if dtype == "float32" and h <= 8 else min(16384, ROWS_MAX // h)
        n = _log_int(rng, 256, longest)
        if rng.random() < 0.4:  # multiples of 128 are as common as other lengths
            n = max(256, n // 128 * 128)
        return _case("op", train, _batch(rng, h, n), h, n, d, dtype, causal=rng.random() < 0.4)
    dtype = rng.choice((half, half, "float32"))
    h = rng.choice((4, 8, 16))
    n = _log_int(rng, 200, min(4096, math.isqrt(SCORES_MAX // h)))
    return _case("op", train, _batch(rng, h, n, 8), h, n, rng.choice((32, 64)), dtype, bias="heads")


def prepare(case, seed):
    """Inputs drawn from N(0, 1) as everywhere in this package's benchmark; a window's relative-position bias has the
    standard deviation of its trunc-normal initialisation, a long dense bias the size of the scores themselves."""
    b, h, n, d = (case[x] for x in "bhnd")
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = getattr(torch, case["dtype"])

    def normal(*shape, dtype=dtype, std=1.0, grad=False):
        t = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)
        if std != 1.0:
            t = t.mul_(std)
        return t.to(dtype).requires_grad_(grad)

    train = case["train"]
    if case["entry"] == "packed":
        inputs = (normal(b, n, 3, h, d, grad=train),)
    else:
        inputs = tuple(normal(b, h, n, d, grad=train) for _ in range(3))
    # (in the hooks the output goes on as [B, N, H*D]: its gradient arrives in that memory order)
    dout = None
    if train:
        dout = normal(b, n, h, d).permute(0, 2, 1, 3) if case["entry"] == "packed" else normal(b, h, n, d)
    bias, kwargs = None, {}
    if case["bias"] == "heads":
        window = n <= WINDOW_TOKENS
        bias = normal(1, h, n, n, dtype=torch.float32, std=0.02 if window else 1.0, grad=train)
        if window:              # the keywords that the Swin hook passes
            kwargs = {"algorithm": "paper_scan", "block_m": 64, "block_n": 64, "q_chunk_size": n}
    return {"case": case, "inputs": inputs, "dout": dout, "bias": bias, "kwargs": kwargs}


def run(state):
    case, inputs, bias, kwargs = state["case"], state["inputs"], state["bias"], state["kwargs"]
    train, causal = case["train"], case["causal"]
    if case["entry"] == "packed":
        out = twopass_attention_qkvpacked(*inputs, bias=bias, is_causal=causal, train=train, **kwargs)
    elif train:
        out = twopass_attention_train(*inputs, bias=bias, is_causal=causal, **kwargs)
    else:
        out = twopass_attention(*inputs, bias=bias, is_causal=causal, **kwargs)
    if not train:
        return out
    wrt = inputs if bias is None else inputs + (bias,)
    return (out.detach(),) + torch.autograd.grad(out, wrt, state["dout"])


def work(case):
    """Bytes: q, k, v (dout) read and out (dq, dk, dv) written once, the bias read and its gradient written once.
    Operations: two contractions of the forward and five of the backward over the admissible (query, key) pairs."""
    b, h, n, d = (case[x] for x in "bhnd")
    pairs = n * (n + 1) // 2 if case["causal"] else n * n
    size = 4 if case["dtype"] == "float32" else 2
    moved = (8 if case["train"] else 4) * b * h * n * d * size
    if case["bias"] != "none":
        moved += (2 if case["train"] else 1) * h * n * n * 4
    return {"bytes": moved, "flops": (14 if case["train"] else 4) * b * h * pairs * d}


def tolerance(case):
    """Relative errors that the data types give: probabilities and score gradients are rounded to the input type before
    the second contraction (2^-9 and 2^-12 on average for bf16 and fp16, several such roundings in a row)."""
    return {"float32": {"rel": 1e-5}, "float16": {"rel": 2e-3}, "bfloat16": {"rel": 1e-2}}[case["dtype"]]
