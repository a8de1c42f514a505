"""The work this library is used for, as measurable cases.

A case is a dict of plain values; `prepare` makes what a program holds before the call (tensors on the GPU, a
layer, a learned bias), `run` makes one call through the public entry points and returns whole outputs: the
attention output (and log-sum-exp) of a forward, and every gradient of a training step.

Kinds of case
  train   flash_attention_v100 forward + backward through autograd (self-attention, Nq == Nk)
  infer   flash_attention_v100 forward without gradients: prompts, decoding and chunked prefill against a
          key/value cache, with the log-sum-exp a cache-merging caller asks for
  bias    a training step with an additive score bias (learned relative positions) or a padding mask as one
  layer   a training step of EnhancedMultiHeadAttention, projections included
"""
import os
import random
import sys

import torch

# the package lies in a folder of its own below the repository's root, the working folder
sys.path.insert(0, os.path.join(os.getcwd(), "flash-attn-v100_b200"))
import flash_attention_v100 as fa  # noqa: E402

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
# floating-point work of the largest listed case (B1 N16384 H32 D128 causal, forward + backward)
MOST_FLOPS = 3.5 * 2 * 32 * 16384 * 16384 * 128
# a drawn case whose kind has dense fp32 arithmetic, a bias or an unusual head size stays a short call
MOST_FLOPS_SMALL = 4.6e10


def _train(name, B, N, H, D, dtype, causal, Hkv=None, dropout=0.0, std=1.0, outliers=0.0):
    case = {"kind": "train", "B": B, "N": N, "H": H, "Hkv": H if Hkv is None else Hkv, "D": D, "dtype": dtype,
            "causal": causal, "dropout": dropout, "std": std, "outliers": outliers}
    return dict(case, name=name) if name else case


def _infer(name, B, Nq, Nk, H, Hkv, D, dtype, mask, ragged=False):
    """mask: "none", "causal" (Nq == Nk) or "bottom_right" (the last query sees the whole cache);
    ragged: every batch entry has its own number of cached keys (key_lengths)."""
    case = {"kind": "infer", "B": B, "Nq": Nq, "Nk": Nk, "H": H, "Hkv": Hkv, "D": D, "dtype": dtype, "mask": mask,
            "ragged": ragged}
    return dict(case, name=name) if name else case


def _bias(name, B, N, H, D, dtype, causal, form):
    """form: "heads" a learned (1, H, N, N) bias that wants its gradient; "padding" a (B, 1, 1, N) mask of -inf."""
    case = {"kind": "bias", "B": B, "N": N, "H": H, "D": D, "dtype": dtype, "causal": causal, "form": form}
    return dict(case, name=name) if name else case


def _layer(name, B, N, heads, D, dtype, masked):
    """masked: a boolean key-padding mask (ragged sentences); else a causal layer."""
    case = {"kind": "layer", "B": B, "N": N, "H": heads, "D": D, "dtype": dtype, "masked": masked}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one short prompt: latency, launches and host work are all there is
        _infer("prompt_fp16_b1_n128", 1, 128, 128, 8, 8, 64, "fp16", "causal"),
        # one token for each of 32 running requests with caches of their own length, grouped heads: a read of the cache
        _infer("decode_bf16_b32_gqa", 32, 1, 4096, 32, 8, 128, "bf16", "none", ragged=True),
        # the next chunk of a long prompt against what is cached, one request, odd lengths
        _infer("chunk_bf16_n700_k8892", 1, 700, 8892, 32, 8, 128, "bf16", "bottom_right"),
        # image-encoder training step: 196 patches and a class token, many short sequences
        _train("train_fp16_b32_n197", 32, 197, 12, 64, "fp16", False),
        # the quick-start shape in fp32
        _train("train_fp32_b2_n1024", 2, 1024, 12, 64, "fp32", True),
        # encoder training in fp16, head size 64
        _train("train_fp16_b8_n2048_d64", 8, 2048, 16, 64, "fp16", False),
        # decoder layer of a 7-billion-parameter model: the headline workload
        _train("train_bf16_b4_n4096_d128", 4, 4096, 32, 128, "bf16", True, std=0.5),
        # long context, some rows of q and k eight times as large
        _train("train_bf16_b1_n16384_d128", 1, 16384, 32, 128, "bf16", True, outliers=0.01),
        # training with attention dropout
        _train("train_bf16_b32_n2048_drop", 32, 2048, 16, 64, "bf16", True, dropout=0.1),
        # head size between the powers of two
        _train("train_bf16_b4_n1024_d96", 4, 1024, 16, 96, "bf16", True),
        # learned relative-position bias with its gradient
        _bias("train_bf16_b8_n512_bias", 8, 512, 12, 64, "bf16", False, "heads"),
        # a whole encoder layer on ragged sentences, boolean padding mask
        _layer("layer_bf16_b16_n1000", 16, 1000, 16, 64, "bf16", True),
    ]


def _log(rng, lo, hi):
    """A whole number, its logarithm spread evenly over [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng: random.Random):
    kind = rng.choice(["train", "train", "train", "decode", "chunk", "prompt", "fp32", "headdim", "bias", "layer"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "train":
        N, D, causal = _log(rng, 64, 16384), rng.choice([64, 128]), rng.random() < 0.6
        group = rng.choice([1, 1, 4])
        H = group * rng.choice([4, 8])
        B = max(1, min(_log(rng, 1, 64), 65536 // N))
        drop = rng.choice([0.0, 0.0, 0.1]) if N <= 4096 else 0.0
        case = _train(None, B, N, H, D, dtype, causal, Hkv=H // group, dropout=drop)
        while work(case)["flops"] > 0.5 * MOST_FLOPS and case["B"] > 1:
            case["B"] -= 1
        while work(case)["flops"] > MOST_FLOPS:
            case["N"] -= 509
        return case
    if kind == "decode":
        group, Hkv, D = rng.choice([1, 4, 8]), rng.choice([2, 4, 8]), rng.choice([64, 128])
        Nq, Nk = rng.choice([1, 1, 1, 2, 5]), _log(rng, 256, 32768)
        B = max(1, min(_log(rng, 1, 64), (1 << 19) // Nk))
        ragged = Nq == 1 and rng.random() < 0.5
        return _infer(None, B, Nq, Nk, group * Hkv, Hkv, D, dtype, "none" if ragged or Nq == 1 else "bottom_right", ragged)
    if kind == "chunk":
        group, Hkv, D = rng.choice([1, 4, 8]), rng.choice([4, 8]), rng.choice([64, 128])
        Nq = _log(rng, 32, 2048)
        return _infer(None, rng.choice([1, 1, 2, 4]), Nq, Nq + _log(rng, 256, 16384), group * Hkv, Hkv, D, dtype, "bottom_right")
    if kind == "prompt":
        N, D = _log(rng, 16, 8192), rng.choice([64, 128])
        return _infer(None, rng.choice([1, 1, 2, 8]), N, N, 8, 8, D, dtype, rng.choice(["causal", "causal", "none"]))
    if kind == "fp32":
        case = _train(None, rng.choice([1, 2, 4]), _log(rng, 64, 2048), rng.choice([4, 8, 12]), rng.choice([64, 64, 128]),
                      "fp32", rng.random() < 0.6)
    elif kind == "headdim":
        case = _train(None, _log(rng, 1, 16), _log(rng, 64, 2048), rng.choice([4, 8, 16]), rng.choice([32, 40, 80, 96]),
                      dtype, rng.random() < 0.6)
    elif kind == "bias":
        case = _bias(None, _log(rng, 1, 16), _log(rng, 64, 1024), rng.choice([4, 8, 12]), rng.choice([64, 128]), dtype,
                     rng.random() < 0.3, rng.choice(["heads", "heads", "padding"]))
    else:
        case = _layer(None, _log(rng, 1, 32), _log(rng, 64, 2048), rng.choice([8, 12, 16]), 64, dtype, rng.random() < 0.6)
        while case["B"] > 1 and case["B"] * case["N"] > 32768:
            case["B"] -= 1
        return case
    while work(case)["flops"] > MOST_FLOPS_SMALL and case["B"] > 1:
        case["B"] -= 1
    while work(case)["flops"] > MOST_FLOPS_SMALL:
        case["N"] -= 61
    return case


def _randn(gen, shape, dtype, std=1.0):
    return (torch.randn(shape, generator=gen, device="cuda") * std).to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    host = random.Random(seed)
    dtype, B, H, D = DTYPES[case["dtype"]], case["B"], case["H"], case["D"]
    state = {"kind": case["kind"]}
    if case["kind"] == "layer":
        E, N = H * D, case["N"]
        rng_before = torch.random.get_rng_state()
        torch.manual_seed(seed)
        layer = fa.EnhancedMultiHeadAttention(E, H, enable_multi_gpu=False)
        torch.random.set_rng_state(rng_before)
        state["layer"] = layer.to(device="cuda", dtype=dtype)
        state["x"] = _randn(gen, (B, N, E), dtype).requires_grad_(True)
        state["g"] = _randn(gen, (B, N, E), dtype)
        state["causal"], state["mask"] = not case["masked"], None
        if case["masked"]:
            lengths = torch.randint(max(1, N // 2), N + 1, (B, 1), generator=gen, device="cuda")
            state["mask"] = torch.arange(N, device="cuda")[None, :] >= lengths      # True hides a key
        return state
    if case["kind"] == "infer":
        Nq, Nk, Hkv = case["Nq"], case["Nk"], case["Hkv"]
        state["q"] = _randn(gen, (B, Nq, H, D), dtype)
        state["k"], state["v"] = (_randn(gen, (B, Nk, Hkv, D), dtype) for _ in range(2))
        state["causal"] = case["mask"] != "none"
        state["alignment"] = "bottom_right" if case["mask"] == "bottom_right" else "top_left"
        state["lengths"] = None
        if case["ragged"]:
            state["lengths"] = torch.randint(max(1, Nk // 2), Nk + 1, (B,), generator=gen, device="cuda", dtype=torch.int32)
        return state
    N, Hkv, std = case["N"], case.get("Hkv", H), case.get("std", 1.0)
    state["q"] = _randn(gen, (B, N, H, D), dtype, std)
    state["k"], state["v"] = (_randn(gen, (B, N, Hkv, D), dtype, std) for _ in range(2))
    if case.get("outliers", 0.0) > 0.0:
        for n in ("q", "k"):
            t = state[n]
            t *= torch.where(torch.rand(t.shape[:3] + (1,), generator=gen, device="cuda") < case["outliers"], 8.0, 1.0).to(dtype)
    for n in ("q", "k", "v"):
        state[n].requires_grad_(True)
    state["g"] = _randn(gen, (B, N, H, D), dtype)
    state["causal"], state["dropout"] = case["causal"], case.get("dropout", 0.0)
    state["stream"] = (host.getrandbits(62), host.getrandbits(30))      # the step's dropout stream
    if case["kind"] == "bias":
        if case["form"] == "heads":
            state["bias"] = _randn(gen, (1, H, N, N), torch.float32, 0.5).requires_grad_(True)
        else:
            lengths = torch.randint(max(1, N // 2), N + 1, (B, 1, 1, 1), generator=gen, device="cuda")
            hidden = torch.arange(N, device="cuda").view(1, 1, 1, N) >= lengths
            state["bias"] = torch.zeros(hidden.shape, device="cuda").masked_fill_(hidden, float("-inf"))
    return state


def run(state):
    kind = state["kind"]
    if kind == "infer":
        with torch.no_grad():
            return fa.flash_attention_v100(state["q"], state["k"], state["v"], causal=state["causal"], return_softmax_lse=True,
                                           key_lengths=state["lengths"], causal_alignment=state["alignment"],
                                           enable_multi_gpu=False)
    if kind == "layer":
        layer, x = state["layer"], state["x"]
        out, _ = layer(x, key_padding_mask=state["mask"], is_causal=state["causal"])
        names, params = zip(*layer.named_parameters())
        grads = torch.autograd.grad(out, (x,) + params, state["g"])
        # the gradient of the key projection's bias is zero but for rounding (softmax ignores a shift of a row)
        return (out,) + tuple(g for n, g in zip(("x",) + names, grads) if n != "k_proj.bias")
    wrt = [state["q"], state["k"], state["v"]]
    if kind == "bias":
        if state["bias"].requires_grad:
            wrt.append(state["bias"])
        out = fa.flash_attention_v100(*wrt[:3], causal=state["causal"], bias=state["bias"], enable_multi_gpu=False)
    else:
        out = fa.flash_attention_v100(*wrt, causal=state["causal"], dropout_p=state["dropout"], enable_multi_gpu=False,
                                      dropout_stream=state["stream"] if state["dropout"] > 0.0 else None)
    return (out,) + torch.autograd.grad(out, wrt, state["g"])


def work(case):
    """Inputs read once, outputs written once; 4 flops per score and head element forward, 10 backward, scores a
    causal mask hides left out."""
    B, H, D, e = case["B"], case["H"], case["D"], 4 if case["dtype"] == "fp32" else 2
    if case["kind"] == "infer":
        Nq, Nk, Hkv = case["Nq"], case["Nk"], case["Hkv"]
        seen = float(Nq * Nk)
        if case["mask"] != "none":
            seen = Nq * (Nk - (Nq - 1) / 2.0)
        keys = 0.75 * Nk if case["ragged"] else Nk              # mean of the drawn key counts
        seen *= keys / Nk
        return {"bytes": e * B * D * (2.0 * Nq * H + 2.0 * keys * Hkv) + 4.0 * B * H * Nq, "flops": 4.0 * B * H * seen * D}
    N = case["N"]
    causal = not case["masked"] if case["kind"] == "layer" else case["causal"]
    seen = N * (N + 1) / 2.0 if causal else float(N * N)
    if case["kind"] == "layer":
        E = H * D
        if case["masked"]:
            seen *= 0.75                                         # mean share of kept keys
        # x, g in and out, dx out; four weights in, their gradients out; four projections, forward and twice backward
        return {"bytes": e * (4.0 * B * N * E + 8.0 * E * E), "flops": 14.0 * B * H * seen * D + 3 * 4 * 2.0 * B * N * E * E}
    Hkv = case.get("Hkv", H)
    # q, k, v, g in; o, dq, dk, dv out
    total = e * B * N * D * (4.0 * H + 4.0 * Hkv)
    if case["kind"] == "bias":
        total += 8.0 * H * N * N if case["form"] == "heads" else 4.0 * B * N
        if case["form"] == "padding":
            seen *= 0.75
    return {"bytes": total, "flops": 14.0 * B * H * seen * D}


def tolerance(case):
    """Four times the error seen against the same call in float64 on the same rounded inputs (listed and drawn cases):
                rel      max (of the result's root mean square, or of the value where that is larger)
        fp16    3.0e-4   1e-2     early causal rows of dq, whose terms cancel
        bf16    1.7e-3   2e-2     the rounding of an exact result alone is 1.6e-3
        fp32    9.3e-6   4e-5
    A layer chains four projections in its own type: 6e-4 and 7e-3 in fp16, 4.8e-3 and 3e-2 in bf16."""
    layer = case["kind"] == "layer"
    return {"fp16": {"rel": 2.5e-3 if layer else 1.2e-3, "max": 0.04}, "bf16": {"rel": 2e-2 if layer else 7e-3, "max": 0.12 if layer else 0.08},
            "fp32": {"rel": 4e-5, "max": 2e-4}}[case["dtype"]]
