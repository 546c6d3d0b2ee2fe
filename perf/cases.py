"""The work a user of the quantized-linear framework has it do, as measurable cases.

Six kinds of layer, each through the public entry point a program calls in steady state:

* ``decode``     one W4A16 projection of a decode step (1..16 tokens) through its bound hot callable
* ``awq``        ``AWQW4A16Linear`` called as a module, whatever the number of tokens
* ``mlp``        the W4A16 SwiGLU MLP block: decode, small batches, chunked and full prefill
* ``w8a8``       ConvRot W8A8 linear: rotation, per-token int8, int8 GEMM
* ``w4a4``       SVDQuant W4A4 linear: rotation, group-64 int4, int4 GEMM, rank-r branch
* ``svdq_w8a8``  SVDQuant W8A8 linear: per-token int8, int8 GEMM, rank-r branch

Weights are made already laid out (what a program does once per layer); a pass is one call on new activations.
"""

import math

import torch

from xqt_b200 import quantize
from xqt_b200.modules import AWQW4A16Linear
from xqt_b200.ops import svdq_w8a8, w4a4, w8a8
from xqt_b200.ops.mlp import W4A16SwiGLUMLP
from xqt_b200.ops.w4a16 import bind_w4a16_decode, prepare_decode

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # the smallest call of a decode step: one token through a key / value projection of an 8B-class decoder
        {"name": "decode_kv_m1", "kind": "decode", "m": 1, "k": 4096, "n": 1024, "group": 128, "dtype": "bf16"},
        # sixteen sequences decoded together through the MLP's down projection
        {"name": "decode_down_m16", "kind": "decode", "m": 16, "k": 14336, "n": 4096, "group": 128, "dtype": "bf16"},
        # a few hundred prompt tokens (a ragged prompt) through an attention projection held as a module, fp16, group 64
        {"name": "awq_prompt_m300", "kind": "awq", "m": 300, "k": 4096, "n": 4096, "group": 64, "dtype": "fp16"},
        # the MLP block of an 8B-class decoder: single-sequence decode, batched decode, a prefill chunk, a full prefill
        {"name": "mlp_m1", "kind": "mlp", "m": 1, "k": 4096, "n": 14336, "group": 128, "dtype": "bf16"},
        {"name": "mlp_m16", "kind": "mlp", "m": 16, "k": 4096, "n": 14336, "group": 128, "dtype": "bf16"},
        {"name": "mlp_m512", "kind": "mlp", "m": 512, "k": 4096, "n": 14336, "group": 128, "dtype": "bf16"},
        {"name": "mlp_m4096", "kind": "mlp", "m": 4096, "k": 4096, "n": 14336, "group": 128, "dtype": "bf16"},
        # a text encoder's 77 tokens through an int8 layer whose width is no multiple of a tile
        {"name": "w8a8_text_m77", "kind": "w8a8", "m": 77, "k": 2048, "n": 5000, "dtype": "fp16", "block": 256, "bias": True},
        # an image's 2048 tokens through an int8 attention projection
        {"name": "w8a8_image_m2048", "kind": "w8a8", "m": 2048, "k": 4096, "n": 4096, "dtype": "bf16", "block": 256, "bias": False},
        # a diffusion transformer (hidden 3072): the MLP's up projection on 4096 image tokens, and an attention projection
        # on a smaller image whose token count is no multiple of a tile
        {"name": "w4a4_dit_m4096", "kind": "w4a4", "m": 4096, "k": 3072, "n": 12288, "dtype": "bf16", "block": 128, "rank": 32, "bias": True},
        {"name": "w4a4_dit_m1000", "kind": "w4a4", "m": 1000, "k": 3072, "n": 3072, "dtype": "fp16", "block": 256, "rank": 16, "bias": True},
        # the int8 layer with a low-rank branch on 2048 tokens
        {"name": "svdq_w8a8_m2048", "kind": "svdq_w8a8", "m": 2048, "k": 4096, "n": 4096, "dtype": "bf16", "rank": 32, "bias": True},
    ]


def _log_int(rng, low, high, step):
    """A multiple of ``step`` in [low, high], spread over the logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high))) / step)) * step))


def draw(rng):
    kind = rng.choice(("decode", "awq", "mlp", "w8a8", "w4a4", "svdq_w8a8"))
    case = {"kind": kind, "dtype": rng.choice(("bf16", "bf16", "fp16"))}
    if kind == "decode":
        case.update(m=rng.randint(1, 16), k=_log_int(rng, 1024, 14336, 128), n=_log_int(rng, 1024, 14336, 8),
                    group=rng.choice((64, 128)))
    elif kind == "awq":
        case.update(m=_log_int(rng, 1, 4096, 1), k=_log_int(rng, 1024, 8192, 128), n=_log_int(rng, 1024, 8192, 8),
                    group=rng.choice((64, 128)))
    elif kind == "mlp":
        case.update(m=_log_int(rng, 1, 4096, 1), k=_log_int(rng, 1024, 4096, 128), n=_log_int(rng, 2816, 14336, 128),
                    group=rng.choice((64, 128, 128)))
    elif kind == "w8a8":
        case.update(m=_log_int(rng, 1, 4096, 1), k=_log_int(rng, 1024, 8192, 256), n=_log_int(rng, 1024, 8192, 8),
                    block=rng.choice((64, 256)), bias=rng.random() < 0.5)
    elif kind == "w4a4":
        case.update(m=_log_int(rng, 16, 4096, 1), k=_log_int(rng, 1024, 3072, 256), n=_log_int(rng, 1024, 12288, 8),
                    block=rng.choice((128, 256)), rank=rng.choice((16, 32)), bias=rng.random() < 0.5)
    else:
        case.update(m=_log_int(rng, 1, 4096, 1), k=_log_int(rng, 1024, 8192, 128), n=_log_int(rng, 1024, 8192, 8),
                    rank=rng.choice((16, 32)), bias=rng.random() < 0.5)
    return case


def _normal(gen, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=gen, device="cuda") * std).to(dtype)


def _activation(gen, m, k, dtype, outliers=False):
    """N(0, 1); ``outliers``: one channel in a hundred twenty times as large, what the rotation is there for."""
    x = _normal(gen, m, k)
    if outliers:
        x[:, torch.randperm(k, generator=gen, device="cuda")[: max(1, k // 100)]] *= 20.0
    return x.to(dtype)


def _low_rank(gen, n, k, rank, dtype):
    """Factors as a truncated SVD of an N(0, 0.02) weight leaves them: Haar directions, singular values at the edge."""
    root = math.sqrt(0.02 * (math.sqrt(n) + math.sqrt(k)))
    return _normal(gen, rank, k, std=root / math.sqrt(k), dtype=dtype), _normal(gen, n, rank, std=root / math.sqrt(n), dtype=dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind, m, k, n, dtype = case["kind"], case["m"], case["k"], case["n"], DTYPES[case["dtype"]]
    bias = _normal(gen, n, std=0.1) if case.get("bias") else None
    if kind in ("decode", "awq", "mlp"):
        def layer(rows, columns):
            return quantize.quantize_w4_asymmetric(_normal(gen, rows, columns, std=0.02), group_size=case["group"],
                                                   param_dtype=dtype, dtype=case["dtype"])

        if kind == "mlp":
            gate, up, down = layer(n, k), layer(n, k), layer(k, n)
            call = W4A16SwiGLUMLP(gate, up, down, device=torch.device("cuda", 0), dtype=dtype)
        elif kind == "awq":
            call = AWQW4A16Linear(layer(n, k)).eval()
        else:
            w = layer(n, k)
            call = bind_w4a16_decode(prepare_decode(w.qweight, w.scales, w.zero_points, group_size=case["group"],
                                                    nibble_signed=False), rows=m, dtype=dtype)
        return {"call": call, "x": _activation(gen, m, k, dtype)}
    weight = _normal(gen, n, k, std=0.02)
    if kind == "w8a8":
        codes, scale = quantize.quantize_w8_per_channel(weight)
        packed = w8a8.pack_convrot_w8a8_linear(codes.t().contiguous(), scale, bias, dtype=dtype)
        call = w8a8.bind_convrot_w8a8_linear(packed, rows=m, rot_size=case["block"])
        return {"call": call, "x": _activation(gen, m, k, dtype, outliers=True)}
    down, up = _low_rank(gen, n, k, case["rank"], dtype)
    if kind == "w4a4":
        codes, scale, _ = quantize.quantize_residual_int4(weight, group_size=64)
        packed = w4a4.pack_svdq_w4a4_linear(None, down, up, bias, packed_residual=codes, residual_scale=scale, dtype=dtype,
                                            rotation=quantize.randomized_rotation(case["block"], seed))
        call = w4a4.bind_svdq_w4a4_linear(packed, rows=m)
        return {"call": call, "x": _activation(gen, m, k, dtype, outliers=True)}
    packed = svdq_w8a8.pack_svdq_w8a8_linear(weight.to(dtype), down, up, bias)
    return {"call": svdq_w8a8.bind_svdq_w8a8_linear(packed, rows=m), "x": _activation(gen, m, k, dtype)}


@torch.no_grad()
def run(state):
    return state["call"](state["x"])


def work(case):
    """Packed weights and their parameters read once, activations read once, outputs written once; the products."""
    kind, m, k, n = case["kind"], case["m"], case["k"], case["n"]
    if kind in ("decode", "awq"):
        return {"bytes": n * k / 2 + 4 * n * k / case["group"] + 2 * m * (k + n), "flops": 2 * m * n * k}
    if kind == "mlp":
        return {"bytes": 3 * (n * k / 2 + 4 * n * k / case["group"]) + 4 * m * k, "flops": 6 * m * n * k}
    if kind == "w8a8":
        return {"bytes": n * k + 4 * n + 2 * m * (k + n), "flops": 2 * m * n * k}
    low_rank = {"bytes": 2 * case["rank"] * (k + n), "flops": 2 * m * case["rank"] * (k + n)}
    if kind == "w4a4":
        return {"bytes": n * k / 2 + n * k / 16 + 2 * m * (k + n) + low_rank["bytes"], "flops": 2 * m * n * k + low_rank["flops"]}
    return {"bytes": n * k + 4 * n + 2 * m * (k + n) + low_rank["bytes"], "flops": 2 * m * n * k + low_rank["flops"]}


def tolerance(case):
    """Sums are fp32 everywhere: what is left is the rounding of the output (two implementations may round the same
    sum apart) and of 16-bit operands; the MLP block rounds three times in a row."""
    rel = {"bf16": 3e-3, "fp16": 8e-4}[case["dtype"]] * (1.7 if case["kind"] == "mlp" else 1.0)
    return {"rel": rel, "max": 10 * rel}
