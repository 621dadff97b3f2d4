"""Timed cases of the verify matmul and the steps beside it, through the package's public interface.

A case is a plain dict; ``kind`` names what a program does with it:

  linear   one projection, the same one in each of ``layers`` layers: y = x . W^T for 1...16 rows
  layer    the projections of a decoder layer as four launches (q+k+v stacked, o, gate and up as a
           gated pair, down) with the two RMS norms ahead of them, ``layers`` layers
  head     the language-model head of a greedy verify step: product and arg-max per row
  exl3     an EXL3 projection (rotate, product, rotate), ``layers`` layers
  gather   embedding rows of a quantized table, by id
  expand   a weight decoded to a dense array (the way of prompts too long for the few-row product)
  host     a list of projections fed from and read back to page-locked host memory in one call

Sizes are those of the 27B-shaped stack and of the small configuration in the benchmark, and generic
ones around them. Every layer has weights of its own; all values are synthetic and come from the seed.
"""
from __future__ import annotations

import math

import torch

from ishizuki_b200.interface import (EXL3Linear, EXL3Tensor, FusedLinear, GGMLKernels, GGMLType, GGUFBlocks,
                                     HostBatch, PackedLinear, rmsNorm)

#: GGML block types: where the fp16 block scales sit and the scale that makes weights of about 0.05
#: (IQ1_M spreads its scale over the top nibbles of its four last words).
BLOCKS = {
    "q2_k": (GGMLType.q2K, (80, 82), 3.4e-3),
    "q4_k": (GGMLType.q4K, (0, 2), 2.0e-4),
    "q6_k": (GGMLType.q6K, (208,), 3.4e-5),
    "iq2_xxs": (GGMLType.iq2Xxs, (0,), 9.0e-4),
    "iq2_xs": (GGMLType.iq2Xs, (0,), 8.2e-4),
    "iq2_s": (GGMLType.iq2S, (0,), 9.0e-4),
    "iq3_xxs": (GGMLType.iq3Xxs, (0,), 3.8e-4),
    "iq3_s": (GGMLType.iq3S, (0,), 3.4e-4),
    "iq1_s": (GGMLType.iq1S, (0,), 6.8e-3),
    "iq1_m": (GGMLType.iq1M, (), 6.4e-3),
    "iq4_xs": (GGMLType.iq4Xs, (0,), 4.2e-5),
}
#: MLX affine packs: bits, group size, scale type, Hadamard block of the input rotation.
PACKS = {
    "affine4_g64": (4, 64, torch.float16, 0),
    "affine4_g32": (4, 32, torch.bfloat16, 0),
    "affine4_g128": (4, 128, torch.float16, 0),
    "affine8_g64": (8, 64, torch.float16, 0),
    "affine2_g64": (2, 64, torch.float16, 0),
    "ternary": (2, 128, torch.bfloat16, 128),
}
#: The formats several weights of which can be stacked into one launch.
STACKED = [f for f in (*BLOCKS, *PACKS) if f != "affine8_g64"]
CODEBOOKS = {"3inst": EXL3Tensor.threeInst, "mcg": EXL3Tensor.mcg, "mul1": EXL3Tensor.mul1}
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
EPS = 1e-6


def listed():
    return [
        # plain decoding, the smallest matrix of a layer: what one call costs
        {"name": "kv_q4k_1", "kind": "linear", "format": "q4_k", "n": 1024, "k": 5120, "rows": 1, "layers": 1},
        # the small affine configuration, a full draft of eight rows
        {"name": "square_affine4_8", "kind": "linear", "format": "affine4_g64", "n": 4096, "k": 4096, "rows": 8, "layers": 8},
        # two decoder layers of the 27B stack in Q4_K: plain decoding and the verify step of eight rows
        {"name": "layers_q4k_1", "kind": "layer", "format": "q4_k", "rows": 1, "layers": 2,
         "hidden": 5120, "q": 6144, "kv": 1024, "inter": 17408},
        {"name": "layers_q4k_8", "kind": "layer", "format": "q4_k", "rows": 8, "layers": 2,
         "hidden": 5120, "q": 6144, "kv": 1024, "inter": 17408},
        # the same layers as ternary packs with rotated inputs, a short draft
        {"name": "layers_ternary_4", "kind": "layer", "format": "ternary", "rows": 4, "layers": 2,
         "hidden": 5120, "q": 6144, "kv": 1024, "inter": 17408},
        # the longest draft through a codebook format, tall inputs
        {"name": "down_iq2xs_16", "kind": "linear", "format": "iq2_xs", "n": 5120, "k": 17408, "rows": 16, "layers": 6},
        # a height that is no multiple of anything, an odd draft
        {"name": "ragged_iq3s_5", "kind": "linear", "format": "iq3_s", "n": 11003, "k": 3840, "rows": 5, "layers": 4},
        # the head of a verify step over the whole vocabulary: the largest weight
        {"name": "head_q6k_8", "kind": "head", "format": "q6_k", "n": 248320, "k": 5120, "rows": 8},
        # trellis-coded gate projections
        {"name": "gate_exl3_8", "kind": "exl3", "bits": 4.0, "codebook": "mul1", "n": 17408, "k": 5120, "rows": 8, "layers": 2},
        # a prompt's embedding rows
        {"name": "embed_q4k_2048", "kind": "gather", "format": "q4_k", "n": 248320, "k": 5120, "rows": 2048, "dtype": "bf16"},
        # a gate projection expanded for a long prompt
        {"name": "expand_q6k", "kind": "expand", "format": "q6_k", "n": 17408, "k": 5120, "dtype": "bf16"},
        # a verify step of four layers whose activations live on the host
        {"name": "host_q4k_8", "kind": "host", "format": "q4_k", "rows": 8, "layers": 4,
         "hidden": 5120, "q": 6144, "kv": 1024, "inter": 17408},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng):
    """Rows of a call: one (plain decoding), a draft of up to eight, a longer one."""
    return rng.choice([1, rng.randint(2, 8), rng.randint(2, 8), rng.randint(9, 16)])


def _wide(rng, hi=20480):
    return 256 * _log(rng, 2, hi // 256)


def draw(rng):
    case = _draw(rng)
    # no dearer than the largest listed case: its bytes, and the weights it decodes (a call of more
    # than eight rows and the formats that are slow to decode count double)
    most = 1.25e9 / (1 + (case.get("rows", 0) > 8)) / (1 if case["kind"] == "head" else 2)
    while work(case)["bytes"] > 1.0e9 or (case["kind"] != "gather" and _weights(case) > most):
        if case.get("layers", 1) > 1:
            case["layers"] -= 1
        elif "inter" in case:
            case["inter"] -= 256
        else:
            case["n"] = case["n"] * 7 // 8 // 128 * 128 + case["n"] % 128 * (case["kind"] != "exl3")
    return case


def _weights(case):
    if "inter" in case:
        return case["layers"] * sum(k * sum(heights) for k, heights in _layer_shapes(case))
    return case.get("layers", 1) * case["n"] * case["k"]


def _draw(rng):
    kind = rng.choices(["linear", "layer", "head", "exl3", "gather", "expand", "host"], [6, 3, 1, 2, 1, 1, 1])[0]
    if kind == "linear":
        return {"kind": kind, "format": rng.choice([*BLOCKS, *PACKS]), "n": _log(rng, 256, 36864), "k": _wide(rng),
                "rows": _rows(rng), "layers": rng.randint(1, 6)}
    if kind in ("layer", "host"):
        hidden = 256 * rng.randint(6, 24)
        return {"kind": kind, "format": rng.choice(STACKED), "rows": _rows(rng), "layers": rng.randint(1, 3), "hidden": hidden,
                "q": 256 * rng.randint(6, 28), "kv": 128 * rng.randint(2, 12), "inter": 256 * int(hidden * rng.uniform(2.5, 3.5) / 256)}
    if kind == "head":
        return {"kind": kind, "format": rng.choice(["q4_k", "q6_k", "iq4_xs", "affine4_g64"]), "n": _log(rng, 32000, 248320),
                "k": 256 * rng.randint(6, 20), "rows": _rows(rng)}
    if kind == "exl3":
        bits = rng.choice([1.5, 2.0, 2.5, 3.0, 3.5, 4.0, 4.0, 5.0, 6.0, 8.0])
        return {"kind": kind, "bits": bits, "codebook": "mul1" if bits % 1 else rng.choice([*CODEBOOKS]),
                "n": 128 * _log(rng, 4, 160), "k": 128 * _log(rng, 4, 140), "rows": _rows(rng), "layers": rng.randint(1, 3)}
    if kind == "gather":
        return {"kind": kind, "format": rng.choice([*BLOCKS]), "n": _log(rng, 32000, 248320), "k": 256 * rng.randint(6, 20),
                "rows": _log(rng, 1, 8192), "dtype": rng.choice([*DTYPES])}
    return {"kind": kind, "format": rng.choice([*BLOCKS]), "n": _log(rng, 256, 20480), "k": _wide(rng, 17408),
            "dtype": rng.choice([*DTYPES])}


# ---- inputs ------------------------------------------------------------------------------------------


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _normal(gen, *shape):
    return torch.randn(shape, device="cuda", generator=gen)


def _blocks(gen, fmt, n, k):
    """[n, k] in blocks of a GGML type: uniform codes, fp16 block scales |N(0, 1)| times the type's own."""
    type_, scales_at, scale = BLOCKS[fmt]
    nb = n * (k // 256)
    out = torch.randint(0, 256, (nb, type_.typeSize), dtype=torch.uint8, device="cuda", generator=gen)
    if scales_at:
        for at in scales_at:
            out[:, at:at + 2] = (_normal(gen, nb, 1).abs() * scale).half().view(torch.uint8)
    else:
        d = (_normal(gen, nb).abs() * scale).half().view(torch.int16).to(torch.int32) & 0xFFFF
        for i in range(4):
            out[:, 49 + 2 * i] = (out[:, 49 + 2 * i] & 0x0F) | (((d >> (4 * i)) & 15) << 4).to(torch.uint8)
    return GGUFBlocks(out.reshape(-1), type_, (n, k))


def _pack(gen, fmt, n, k):
    """An affine pack [n, k]: (codes, scales, biases); ternary: codes 0, 1, 2 with bias = -scale."""
    bits, group, dtype, _ = PACKS[fmt]
    if fmt == "ternary":
        u = torch.rand((n, k // 16, 16), device="cuda", generator=gen)
        codes = (u >= 0.3).to(torch.int32) + (u >= 0.7).to(torch.int32)
        words = torch.zeros((n, k // 16), dtype=torch.int32, device="cuda")
        for i in range(16):
            words |= codes[:, :, i] << (2 * i)
        scales = (_normal(gen, n, k // group).abs() * 0.02).to(dtype)
        return words, scales, -scales
    words = torch.randint(-(1 << 31), 1 << 31, (n, k * bits // 32), dtype=torch.int32, device="cuda", generator=gen)
    scales = _normal(gen, n, k // group).abs() * (0.16 / (1 << bits))
    biases = (scales * -(1 << (bits - 1)) + _normal(gen, n, k // group) * 1e-3).to(dtype)
    return words, scales.to(dtype), biases


def _weight(gen, fmt, n, k):
    return _blocks(gen, fmt, n, k) if fmt in BLOCKS else _pack(gen, fmt, n, k)


def _projection(gen, fmt, k, heights, gated=False):
    parts = [_weight(gen, fmt, n, k) for n in heights]
    if fmt in BLOCKS:
        return FusedLinear(parts, gated=gated) if len(parts) > 1 else PackedLinear(ggml=parts[0])
    bits, group, _, block = PACKS[fmt]
    if len(parts) > 1:
        return FusedLinear(parts, None, block, groupSize=group, bits=bits, gated=gated)
    return PackedLinear(*parts[0], None, block, groupSize=group, bits=bits)


def _exl3(gen, case):
    n, k = case["n"], case["k"]
    trellis = torch.randint(-32768, 32768, (k // 16, n // 16, int(16 * case["bits"])), dtype=torch.int16, device="cuda", generator=gen)
    su = torch.where(_normal(gen, k) < 0, -1.0, 1.0).half()
    sv = (torch.where(_normal(gen, n) < 0, -1.0, 1.0) * (0.01 + 0.03 * torch.rand(n, device="cuda", generator=gen))).half()
    return EXL3Linear(EXL3Tensor(trellis, su, sv, CODEBOOKS[case["codebook"]]))


def _layer_shapes(case):
    """(input width, heights) of a layer's four launches: q+k+v, o, gate+up, down."""
    h, q, kv, inter = case["hidden"], case["q"], case["kv"], case["inter"]
    return [(h, (q, kv, kv)), (q, (h,)), (h, (inter, inter)), (inter, (h,))]


def prepare(case, seed):
    gen = _generator(seed)
    kind, rows = case["kind"], case.get("rows", 0)
    if kind in ("linear", "head"):
        lins = [_projection(gen, case["format"], case["k"], (case["n"],)) for _ in range(case.get("layers", 1))]
        return kind, lins, [_normal(gen, rows, case["k"]).half() for _ in lins]
    if kind == "exl3":
        lins = [_exl3(gen, case) for _ in range(case["layers"])]
        return kind, lins, [_normal(gen, rows, case["k"]).half() for _ in lins]
    if kind == "layer":
        layers = []
        for _ in range(case["layers"]):
            qkv, o, gate_up, down = (_projection(gen, case["format"], k, heights, gated=i == 2)
                                     for i, (k, heights) in enumerate(_layer_shapes(case)))
            norms = [(1.0 + 0.1 * _normal(gen, case["hidden"])).half() for _ in range(2)]
            # the residual stream ahead of the attention and of the MLP, and what the attention gives
            inputs = [_normal(gen, rows, case["hidden"]) * 4, _normal(gen, rows, case["q"]).half(), _normal(gen, rows, case["hidden"]) * 4]
            layers.append((qkv, o, gate_up, down, norms, inputs))
        return kind, layers
    if kind == "host":
        lins, xs, ys = [], [], []
        for _ in range(case["layers"]):
            for k, heights in _layer_shapes(case):
                lins.append(_projection(gen, case["format"], k, heights))
                xs.append(_normal(gen, rows, k).half().cpu().pin_memory())
                ys.append(torch.zeros((rows, sum(heights)), dtype=torch.float16).pin_memory())
        return kind, HostBatch(lins, xs, ys)
    w = _blocks(gen, case["format"], case["n"], case["k"])
    dtype = DTYPES[case["dtype"]]
    if kind == "gather":
        return kind, torch.randint(0, case["n"], (rows,), dtype=torch.int32, device="cuda", generator=gen), w, dtype
    return kind, w, dtype


def run(state):
    kind = state[0]
    if kind in ("linear", "exl3"):
        return [lin(x) for lin, x in zip(state[1], state[2])]
    if kind == "head":
        return [lin.argmax(x) for lin, x in zip(state[1], state[2])]
    if kind == "layer":
        out = []
        for qkv, o, gate_up, down, norms, (residual, attention, residual2) in state[1]:
            heads = qkv(rmsNorm(residual, norms[0], EPS))
            mixed = o(attention)
            hidden = gate_up(rmsNorm(residual2, norms[1], EPS))
            out += [heads, mixed, hidden, down(hidden)]
        return out
    if kind == "host":
        batch = state[1]
        batch.run()
        torch.cuda.current_stream().synchronize()  # the outputs are read on the host
        return batch.ys
    if kind == "gather":
        _, ids, w, dtype = state
        return GGMLKernels.gather(ids, w.bytes, w.type, w.inputDim, dtype)
    _, w, dtype = state
    return GGMLKernels.dequantize(w.bytes, w.type, w.shape, dtype)


# ---- what a pass needs ---------------------------------------------------------------------------------


def _row_bytes(fmt, k):
    """Bytes of one output row of a weight."""
    if fmt in BLOCKS:
        return k // 256 * BLOCKS[fmt][0].typeSize
    bits, group, _, _ = PACKS[fmt]
    return k * bits // 8 + 2 * 2 * (k // group)


def work(case):
    kind, layers = case["kind"], case.get("layers", 1)
    n, k, rows = case.get("n", 0), case.get("k", 0), case.get("rows", 0)
    if kind in ("linear", "head"):
        out = 4 * rows if kind == "head" else 2 * rows * n
        return {"bytes": layers * (n * _row_bytes(case["format"], k) + 2 * rows * k + out), "flops": 2.0 * layers * rows * n * k}
    if kind == "exl3":
        return {"bytes": layers * (n * k * case["bits"] / 8 + 2 * (n + k) + 2 * rows * (n + k)), "flops": 2.0 * layers * rows * n * k}
    if kind in ("layer", "host"):
        nbytes, flops = 0, 0.0
        for i, (width, heights) in enumerate(_layer_shapes(case)):
            tall = sum(heights)
            nbytes += tall * _row_bytes(case["format"], width) + 2 * rows * (tall // 2 if kind == "layer" and i == 2 else tall)
            flops += 2.0 * rows * tall * width
            if kind == "host" or i == 1:
                nbytes += 2 * rows * width
            elif i != 3:  # fp32 residual rows and the norm's weight; down reads what gate and up gave
                nbytes += 4 * rows * width + 2 * width
        return {"bytes": layers * nbytes, "flops": layers * flops}
    size = 4 if case["dtype"] == "f32" else 2
    if kind == "gather":
        return {"bytes": rows * (_row_bytes(case["format"], k) + k * size + 4), "flops": 2.0 * rows * k}
    return {"bytes": n * (_row_bytes(case["format"], k) + k * size), "flops": 2.0 * n * k}


def tolerance(case):
    if case["kind"] in ("gather", "expand"):
        return "exact"  # one rounding of an exact value
    if case["kind"] == "head":
        return {"rel": 0.0, "differ": 0.01}  # fp16 logits that tie
    # fp32 sums in another order, then fp16 outputs (eps 4.9e-4); the chained ones round several times
    return {"rel": 1e-3, "max": 1e-2}
