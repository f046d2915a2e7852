"""The work a program has this framework do, as cases that can be timed: `chill_attention()` forward calls and training
steps (forward + gradients of q, k and v) over the range of shapes, masks, data types and options it serves.

    listed()              the cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   tensors and mask object a program holds before the call
    run(state)            one pass through the public call (and autograd)
    work(case)            bytes and floating-point operations a pass cannot do without
    tolerance(case)       how far two correct implementations of the same precision may differ

Import it with the repository's root as the working folder.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "chill-attention_b200"))

import chill_attention as ca  # noqa: E402

_DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
#: mask name -> (class, names of its constants in a case)
_MASKS = {
    "full": (ca.FullChillMask, ()),
    "causal": (ca.CausalChillMask, ()),
    "window": (ca.SlidingWindowChillMask, ("left", "right")),
    "chunkwise": (ca.ChunkwiseChillMask, ("context", "back")),
    "prefix_lm": (ca.PrefixLMChillMask, ("prefix",)),
}


def _case(name, step, mask, dtype, B, H, L, D, kv_heads=None, lens=False, layout="bhld", precision="ieee", **constants):
    c = {"step": step, "mask": mask, "dtype": dtype, "B": B, "H": H, "kv_heads": kv_heads or H, "L": L, "D": D, "lens": lens,
         "layout": layout, "precision": precision, **constants}
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # One layer of a short request or a small encoder: a single wave of tiles, all latency.
        _case("short_forward_fp16", "forward", "full", "fp16", 8, 4, 128, 128),
        # A unit-test or debugging sized training step in the default fp32 precision.
        _case("short_train_fp32", "train", "causal", "fp32", 1, 2, 128, 64),
        # Prefill of a batch of prompts of different lengths: grouped-query heads, tensors as the projections leave them
        # ([batch, position, head, channel] in memory), no gradients.
        _case("prefill_gqa_bf16", "forward", "causal", "bf16", 4, 32, 3000, 128, kv_heads=8, lens=True, layout="blhd"),
        # Local attention with a narrow band over a length that is no multiple of any tile (speech / audio encoders).
        _case("train_narrow_window_fp16", "train", "window", "fp16", 8, 12, 2085, 64, left=16, right=16),
        # Pre-training of a causal decoder, the ordinary large step.
        _case("train_causal_bf16", "train", "causal", "bf16", 8, 16, 4096, 128),
        # Streaming (chunk-by-chunk) encoder on long recordings: short key ranges, head dim 64, memory-heavy.
        _case("train_chunkwise_fp16", "train", "chunkwise", "fp16", 4, 32, 16384, 64, context=128, back=2),
        # Prefix language model: bidirectional prompt, causal continuation.
        _case("train_prefix_lm_bf16", "train", "prefix_lm", "bf16", 4, 16, 8192, 128, prefix=1024),
        # Long-context sliding window, the largest step.
        _case("train_long_window_bf16", "train", "window", "bf16", 1, 32, 131072, 128, left=1024, right=0),
        # fp32 training with the tensor cores allowed to round to TF32.
        _case("train_causal_tf32", "train", "causal", "fp32", 2, 16, 4096, 128, precision="tf32"),
        # fp32 training in the default (IEEE) precision at an ordinary size.
        _case("train_full_fp32", "train", "full", "fp32", 2, 8, 1000, 64),
        # Wide heads.
        _case("train_wide_head_bf16", "train", "causal", "bf16", 2, 16, 4096, 256),
        # Narrow heads of a small model, ragged batch.
        _case("train_narrow_head_fp16", "train", "causal", "fp16", 8, 8, 1024, 32, lens=True, layout="blhd"),
    ]


def _log_int(rng, lo, hi):
    """Whole number from [lo, hi], spread over the logarithm; half of the time rounded to a multiple of 64, where one is near."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if n >= 128 and rng.random() < 0.5:
        n = n // 64 * 64
    return min(max(n, lo), hi)


def _draw_mask(rng, L):
    mask = rng.choice(list(_MASKS))
    if mask == "window":
        left = _log_int(rng, 8, max(16, min(2048, L)))
        return mask, {"left": left, "right": rng.choice([0, left, _log_int(rng, 4, 64)])}
    if mask == "chunkwise":
        return mask, {"context": _log_int(rng, 8, max(16, min(512, L))), "back": rng.randint(0, 8)}
    if mask == "prefix_lm":
        return mask, {"prefix": _log_int(rng, 4, max(8, L // 2))}
    return mask, {}


def draw(rng):
    family = rng.choice(["forward", "forward", "train", "train", "train", "train_head", "train_wide", "train_fp32", "train_tf32"])
    step, precision, kv_groups = ("forward" if family == "forward" else "train"), "ieee", rng.choice([1, 1, 1, 2, 4])
    dtype = rng.choice(["fp16", "bf16"])
    if family in ("forward", "train"):
        D, L = rng.choice([64, 128, 128]), _log_int(rng, 100, 32768 if family == "forward" else 65536)
        most_flops, most_tokens = 5e12, 2 ** 22  # of one pass; tokens = B * H * L
    elif family == "train_head":
        D, L, most_flops, most_tokens = rng.choice([16, 32, 32]), _log_int(rng, 100, 8192), 2e11, 2 ** 18
    elif family == "train_wide":
        D, L, most_flops, most_tokens = 256, _log_int(rng, 100, 8192), 1.5e12, 2 ** 18
    elif family == "train_fp32":
        dtype, D, L, most_flops, most_tokens = "fp32", rng.choice([32, 64, 64, 128]), _log_int(rng, 64, 2048), 8e9, 2 ** 16
    else:
        dtype, precision, D, L, most_flops, most_tokens = "fp32", "tf32", rng.choice([64, 128]), _log_int(rng, 128, 8192), 1e12, 2 ** 18
    mask, constants = _draw_mask(rng, L)
    kv_heads = rng.choice([1, 2, 3, 4, 8])
    c = _case(None, step, mask, dtype, rng.choice([1, 2, 3, 4, 8]), kv_heads * kv_groups, L, D, kv_heads=kv_heads,
              lens=rng.random() < 0.3, layout=rng.choice(["bhld", "blhd"]), precision=precision, **constants)
    while (work(c)["flops"] > most_flops or c["B"] * c["H"] * L > most_tokens) and c["B"] > 1:
        c["B"] //= 2
    while (work(c)["flops"] > most_flops or c["B"] * c["H"] * L > most_tokens) and c["H"] > 1:
        if c["kv_heads"] > 1:
            c["kv_heads"] //= 2
        c["H"] = max(c["kv_heads"], c["H"] // 2 // c["kv_heads"] * c["kv_heads"])
    while work(c)["flops"] > most_flops:
        c["L"] = c["L"] * 3 // 4
    return c


def _mask(case):
    cls, names = _MASKS[case["mask"]]
    return cls(*(case[n] for n in names))


def _lengths(case):
    """Valid lengths of the batch rows: one full row, the rest spread over the upper three quarters of L."""
    B, L = case["B"], case["L"]
    return [max(1, L - (3 * L * i) // (4 * B)) for i in range(B)] if case["lens"] else [L] * B


def prepare(case, seed):
    dev, dtype = torch.device("cuda"), _DTYPES[case["dtype"]]
    g = torch.Generator(device=dev).manual_seed(seed)
    train = case["step"] == "train"

    def tensor(heads):
        B, L, D = case["B"], case["L"], case["D"]
        if case["layout"] == "blhd":
            return torch.randn(B, L, heads, D, generator=g, device=dev, dtype=dtype).transpose(1, 2)
        return torch.randn(B, heads, L, D, generator=g, device=dev, dtype=dtype)

    q, k, v = tensor(case["H"]), tensor(case["kv_heads"]), tensor(case["kv_heads"])
    state = {"q": q, "k": k, "v": v, "mask": _mask(case), "lens": None, "precision": case["precision"]}
    if case["lens"]:
        order = torch.randperm(case["B"], generator=torch.Generator().manual_seed(seed))
        state["lens"] = torch.tensor(_lengths(case), dtype=torch.int32)[order].to(dev)
    if train:
        state["do"] = tensor(case["H"])
        for t in (q, k, v):
            t.requires_grad_(True)
    return state


def run(state):
    q, k, v = state["q"], state["k"], state["v"]
    if "do" not in state:
        return ca.chill_attention(q, k, v, mask=state["mask"], lens=state["lens"], precision=state["precision"])
    o = ca.chill_attention(q, k, v, mask=state["mask"], lens=state["lens"], precision=state["precision"])
    dq, dk, dv = torch.autograd.grad(o, (q, k, v), state["do"])
    return o.detach(), dq, dk, dv


def _pairs(mask, L):
    """Visible (query, key) pairs of one head and batch row (every mask's rows are one key interval)."""
    q = np.arange(L, dtype=np.int64)
    lo, hi = type(mask).k_range_for_q(torch.from_numpy(q), L, mask.constargs)
    lo = torch.as_tensor(lo).expand(L).clamp(min=0)
    hi = torch.as_tensor(hi).expand(L).clamp(max=L - 1)
    return int((hi - lo + 1).clamp(min=0).sum())


def work(case):
    mask, train = _mask(case), case["step"] == "train"
    pairs = sum(_pairs(mask, n) for n in _lengths(case)) * case["H"]
    # q, o and k, v once each; a training step also reads the incoming gradient and writes three
    rows = case["B"] * case["L"] * (case["H"] * (4 if train else 2) + case["kv_heads"] * (4 if train else 2))
    return {"bytes": rows * case["D"] * _DTYPES[case["dtype"]].itemsize,
            "flops": pairs * case["D"] * (14 if train else 4)}


def tolerance(case):
    # About four times the distance from the same computation in 64 bits, which is (largest of O, dQ, dK, dV; rel / max):
    # bf16 3.0e-3 / 0.13 (8-bit mantissa of results and probabilities), fp16 3.8e-4 / 0.012, TF32 1.8e-3 / 0.04 (11-bit
    # products), fp32 7.3e-7 / 7e-6 (order of the sums).
    if case["precision"] == "tf32":
        return {"rel": 7e-3, "max": 0.16}
    return {"fp32": {"rel": 4e-6, "max": 4e-5}, "fp16": {"rel": 1.6e-3, "max": 0.05}, "bf16": {"rel": 1.2e-2, "max": 0.5}}[case["dtype"]]
