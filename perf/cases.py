"""What this framework is timed on: weight-only quantized linears as an inference engine runs them.

A case is a dict of plain values; its ``kind`` says which of the public entry points it goes through.

* ``step``: the projections of one or more decoder layers, installed on the model's modules by
  ``install_w4a16`` / ``quantize_linear_modules`` (and, with ``fused``, ``install_fused_qkv`` /
  ``install_fused_swiglu``).  With ``graph`` the step is captured once and replayed, which is how an
  engine runs decode and mixed steps; without it the modules are called eagerly, which is how it runs
  prefill chunks.  ``tokens`` is the number of activation rows: decode batch, mixed step or prompt
  chunk.  Attention itself, norms and the residual stream are not part of the framework: every
  projection is fed activations of its own.
* ``linear``: one call of the functional API (``w4a16_linear`` / ``w8a16_linear``), eager.
* ``w8a8``: ``w8a8_linear`` over the projections of a layer (large prompts), eager.
* ``load``: quantize-on-load of a layer's weights (the encode direction), eager.
* ``dequant``: ``w4_dequantize_into`` (the decode direction), eager.

Formats: ``w8`` int8 per channel, ``w4`` the group-128 split-half layout, ``w4z`` group-128 with
zero-points.  Weights are N(0, 0.02) and activations N(0, 1), one per cent of the rows of a large
prompt scaled by 20 as outliers.
"""

from __future__ import annotations

import math

import torch
from torch import nn

from full_inference_engine_b200.kernels import w4a16_format as w4_format
from full_inference_engine_b200.kernels import w4a16_linear as w4_kernels
from full_inference_engine_b200.kernels import w8a16_linear as w8_kernels
from full_inference_engine_b200.kernels import w8a8_linear as w8a8_kernels
from full_inference_engine_b200.quantization.fused_mlp import install_fused_swiglu
from full_inference_engine_b200.quantization.fused_qkv import install_fused_qkv
from full_inference_engine_b200.quantization.int8 import quantize_linear_modules
from full_inference_engine_b200.quantization.w4a16 import install_w4a16

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
LARGEST_FLOPS = 4.1e11        # of one pass: 4096 tokens through 4096 -> 12288 (16-bit operands)
LARGEST_INT8_OPS = 6.3e11     # 4096 tokens through the layer of the int8 x int8 case
LARGEST_WEIGHTS = 4.0e8       # bytes of quantized weights of one pass


def step(name, fmt, dtype, tokens, layers, hidden, q, kv, ffn, *, fused, graph, bias=False):
    return {"name": name, "kind": "step", "fmt": fmt, "dtype": dtype, "tokens": tokens, "layers": layers,
            "hidden": hidden, "q": q, "kv": kv, "ffn": ffn, "fused": fused, "graph": graph, "bias": bias}


def listed():
    qwen3_8b = dict(hidden=4096, q=4096, kv=1024, ffn=12288)
    qwen3_0_6b = dict(hidden=1024, q=2048, kv=1024, ffn=3072)
    qwen25_3b = dict(hidden=2048, q=2048, kv=256, ffn=11008)
    return [
        # the smallest call: one int8 projection of a small model at a decode batch of 8, eager, where
        # the host path and one short launch are everything
        {"name": "w8_call_b8", "kind": "linear", "fmt": "w8", "dtype": "fp16", "tokens": 8, "k": 1024,
         "n": 3072, "bias": False},
        # one user at a time: single-token decode steps of 4-bit and int8 8B-shaped layers
        step("w4_decode_b1", "w4", "bf16", 1, 3, **qwen3_8b, fused=True, graph=True),
        step("w8_decode_b1", "w8", "bf16", 1, 2, **qwen3_8b, fused=False, graph=True),
        # continuous batching: a moderate and a large decode batch, the large one an odd count
        step("w4_decode_b16", "w4", "fp16", 16, 3, **qwen3_8b, fused=True, graph=True),
        step("w8_decode_b61", "w8", "bf16", 61, 2, **qwen3_8b, fused=True, graph=True),
        # speculative or very large batches on 4-bit weights, projections not fused
        step("w4_decode_b40", "w4", "bf16", 40, 2, **qwen3_8b, fused=False, graph=True),
        # a mixed step of a small model: 16 decode rows and a 128-token chunk
        step("w8_mixed_m144", "w8", "fp16", 144, 8, **qwen3_0_6b, fused=False, graph=True),
        # an odd prompt chunk through 4-bit layers with biases, eager
        step("w4_prefill_m777", "w4", "fp16", 777, 1, **qwen25_3b, fused=True, graph=False, bias=True),
        # a full prompt through zero-point 4-bit weights: the tensor-bound end of the range
        {"name": "w4z_prefill_m4096", "kind": "linear", "fmt": "w4z", "dtype": "bf16", "tokens": 4096,
         "k": 4096, "n": 12288, "bias": False},
        # the output head at a decode batch (its logits feed a sampler): the largest matrix
        {"name": "w4_head_b16", "kind": "linear", "fmt": "w4", "dtype": "fp16", "tokens": 16, "k": 4096,
         "n": 151936, "bias": False},
        # a full prompt through the int8 x int8 path
        {"name": "w8a8_prefill_m4096", "kind": "w8a8", "dtype": "fp16", "tokens": 4096, "hidden": 2048,
         "q": 2048, "kv": 256, "ffn": 11008},
        # loading: a layer's bf16 weights become 4-bit
        {"name": "w4_load_layer", "kind": "load", "fmt": "w4", "dtype": "bf16", "hidden": 4096, "q": 4096,
         "kv": 1024, "ffn": 12288},
    ]


# ------------------------------------------------------------------------------ drawn cases
def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _multiple(rng, low, high, of):
    return max(1, round(_log_int(rng, low, high) / of)) * of


def _layer_shape(rng):
    hidden = _multiple(rng, 1024, 4096, 128)
    kv = rng.choice([hidden, hidden // 4, max(128, hidden // 8)])
    q = rng.choice([hidden, 2 * hidden if hidden <= 2048 else hidden])
    return {"hidden": hidden, "q": q, "kv": max(32, kv // 32 * 32), "ffn": _multiple(rng, 2.5 * hidden, 5.4 * hidden, 128)}


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "mixed", "prefill", "linear", "linear", "head", "w8a8", "load",
                       "dequant"])
    dtype = rng.choice(["fp16", "bf16"])
    if kind in ("decode", "mixed", "prefill"):
        shape = _layer_shape(rng)
        fmt = rng.choice(["w4", "w8"])
        fused = rng.choice([True, True, False])
        tokens = {"decode": _log_int(rng, 1, 64), "mixed": rng.randint(65, 256),
                  "prefill": _log_int(rng, 257, 4096)}[kind]
        case = {"kind": "step", "fmt": fmt, "dtype": dtype, "tokens": tokens, "layers": 1, **shape, "fused": fused,
                "graph": kind != "prefill", "bias": rng.choice([False, False, True])}
        one = work(case)
        if kind != "prefill":
            case["layers"] = max(1, min(8, int(LARGEST_WEIGHTS / one["bytes"])))
        elif one["flops"] > LARGEST_FLOPS:
            case["tokens"] = max(257, int(tokens * LARGEST_FLOPS / one["flops"]))
        return case
    if kind == "linear":
        fmt = rng.choice(["w8", "w4", "w4z"])
        k = _multiple(rng, 1024, 12288, 128)
        n = _log_int(rng, 512, 16384)
        tokens = _log_int(rng, 1, 4096)
        tokens = max(1, min(tokens, int(LARGEST_FLOPS / (2.0 * k * n))))
        return {"kind": "linear", "fmt": fmt, "dtype": dtype, "tokens": tokens, "k": k, "n": n,
                "bias": rng.choice([False, True])}
    if kind == "head":
        return {"kind": "linear", "fmt": rng.choice(["w4", "w8"]), "dtype": dtype, "tokens": _log_int(rng, 1, 64),
                "k": _multiple(rng, 1024, 4096, 128), "n": _log_int(rng, 32000, 151936), "bias": False}
    if kind == "w8a8":
        case = {"kind": "w8a8", "dtype": dtype, "tokens": _log_int(rng, 65, 4096), **_layer_shape(rng)}
        case["tokens"] = min(case["tokens"], int(case["tokens"] * LARGEST_INT8_OPS / work(case)["flops"]))
        return case
    shape = _layer_shape(rng)
    if kind == "load":
        return {"kind": "load", "fmt": rng.choice(["w4", "w8", "w4z"]), "dtype": rng.choice(["bf16", "bf16", "fp32"]),
                **shape}
    return {"kind": "dequant", "fmt": rng.choice(["w4", "w4z"]), "n": _log_int(rng, 1024, 12288),
            "k": _multiple(rng, 1024, 12288, 128)}


# ------------------------------------------------------------------------------ inputs and weights
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _weight(gen, n, k, dtype):
    return torch.randn(n, k, generator=gen, device="cuda", dtype=dtype) * 0.02


def _activations(gen, tokens, width, dtype):
    x = torch.randn(tokens, width, generator=gen, device="cuda")
    if tokens >= 256:
        rows = torch.randperm(tokens, generator=gen, device="cuda")[: max(1, tokens // 100)]
        x[rows] *= 20.0
    return x.to(dtype)


def _linear(gen, k, n, dtype, bias):
    linear = torch.nn.utils.skip_init(nn.Linear, k, n, bias=bias, device="cuda", dtype=dtype)
    linear.weight.data.copy_(_weight(gen, n, k, dtype))
    if bias:
        linear.bias.data.copy_(torch.randn(n, generator=gen, device="cuda") * 0.1)
    return linear


class Attention(nn.Module):
    def __init__(self, gen, case, dtype):
        super().__init__()
        hidden, q, kv, bias = case["hidden"], case["q"], case["kv"], case["bias"]
        self.q_proj = _linear(gen, hidden, q, dtype, bias)
        self.k_proj = _linear(gen, hidden, kv, dtype, bias)
        self.v_proj = _linear(gen, hidden, kv, dtype, bias)
        self.o_proj = _linear(gen, q, hidden, dtype, False)


class FeedForward(nn.Module):
    def __init__(self, gen, case, dtype):
        super().__init__()
        self.gate_proj = _linear(gen, case["hidden"], case["ffn"], dtype, False)
        self.up_proj = _linear(gen, case["hidden"], case["ffn"], dtype, False)
        self.down_proj = _linear(gen, case["ffn"], case["hidden"], dtype, False)

    def forward(self, hidden_states):
        return self.down_proj(nn.functional.silu(self.gate_proj(hidden_states)) * self.up_proj(hidden_states))


class Layer(nn.Module):
    def __init__(self, gen, case, dtype):
        super().__init__()
        self.self_attn = Attention(gen, case, dtype)
        self.mlp = FeedForward(gen, case, dtype)


def _layer_outputs(layer, fused, inputs):
    """Every projection of a layer, as its model code calls them."""
    hidden, context, mlp_in, mlp_mid = inputs
    attention, mlp = layer.self_attn, layer.mlp
    outputs = [attention.q_proj(hidden), attention.k_proj(hidden), attention.v_proj(hidden), attention.o_proj(context)]
    if fused:
        outputs.append(mlp(mlp_in))
    else:
        outputs += [mlp.gate_proj(mlp_in), mlp.up_proj(mlp_in), mlp.down_proj(mlp_mid)]
    return outputs


def _prepare_step(case, seed):
    gen = _generator(seed)
    dtype = DTYPES[case["dtype"]]
    layers = nn.ModuleList()
    for _ in range(case["layers"]):
        layer = Layer(gen, case, dtype)
        if case["fmt"] == "w4":
            install_w4a16(layer)
        else:
            quantize_linear_modules(layer)
        if case["fused"]:
            install_fused_qkv(layer)
            install_fused_swiglu(layer)
        layers.append(layer)
    tokens = case["tokens"]
    inputs = [[_activations(gen, tokens, case["hidden"], dtype), _activations(gen, tokens, case["q"], dtype),
               _activations(gen, tokens, case["hidden"], dtype),
               None if case["fused"] else _activations(gen, tokens, case["ffn"], dtype)] for _ in layers]

    def forward():
        with torch.no_grad():
            return [y for layer, xs in zip(layers, inputs) for y in _layer_outputs(layer, case["fused"], xs)]

    if not case["graph"]:
        return {"forward": forward}
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        forward()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outputs = forward()
    return {"graph": graph, "outputs": outputs, "keep": (layers, inputs)}


def _quantize(fmt, weight):
    if fmt == "w8":
        return w8_kernels.quantize_weight_per_channel(weight)
    if fmt == "w4":
        return w4_format.quantize_weight_w4_grouped(weight)
    return w4_format.quantize_weight_w4_asym(weight)


def _layer_matrices(case):
    """(n, k) of a layer's projections, those that read the same activations as one matrix."""
    return [(case["q"] + 2 * case["kv"], case["hidden"]), (case["hidden"], case["q"]),
            (2 * case["ffn"], case["hidden"]), (case["hidden"], case["ffn"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _prepare_step(case, seed)
    gen = _generator(seed)
    dtype = DTYPES[case.get("dtype", "fp16")]
    if kind == "linear":
        n, k = case["n"], case["k"]
        weights = _quantize(case["fmt"], _weight(gen, n, k, dtype))
        x = _activations(gen, case["tokens"], k, dtype)
        bias = (torch.randn(n, generator=gen, device="cuda") * 0.1).to(dtype) if case["bias"] else None
        if case["fmt"] == "w8":
            return {"forward": lambda: w8_kernels.w8a16_linear(x, weights[0], weights[1], bias, static_weights=True)}
        zeros = weights[2] if case["fmt"] == "w4z" else None
        return {"forward": lambda: w4_kernels.w4a16_linear(x, weights[0], weights[1], bias, zeros=zeros,
                                                           static_weights=True)}
    if kind == "w8a8":
        calls = []
        for n, k in _layer_matrices(case):
            q, scales = w8_kernels.quantize_weight_per_channel(_weight(gen, n, k, dtype))
            calls.append((_activations(gen, case["tokens"], k, dtype), w8a8_kernels.pack_w8a8_weight(q), scales))
        return {"forward": lambda: [w8a8_kernels.w8a8_linear(*call) for call in calls]}
    if kind == "load":
        weights = [_weight(gen, n, k, dtype) for n, k in _layer_matrices(case)]
        return {"forward": lambda: [_quantize(case["fmt"], w) for w in weights]}
    n, k = case["n"], case["k"]
    weights = _quantize(case["fmt"], _weight(gen, n, k, torch.bfloat16))
    out = torch.empty(n, k, dtype=torch.float16, device="cuda")
    zeros = weights[2] if case["fmt"] == "w4z" else None
    return {"forward": lambda: w4_kernels.w4_dequantize_into(out, weights[0], weights[1], zeros=zeros)}


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["outputs"]
    return state["forward"]()


# ------------------------------------------------------------------------------ what a pass needs
def _weight_bytes(fmt, n, k, scale_bytes=2):
    if fmt == "w8":
        return n * k + scale_bytes * n
    return n * k // 2 + (2 if fmt == "w4" else 4) * n * (k // 128)


def work(case):
    kind = case["kind"]
    if kind == "step":
        m = case["tokens"]
        hidden, q, kv, ffn, fused = case["hidden"], case["q"], case["kv"], case["ffn"], case["fused"]
        shapes = [(q, hidden), (kv, hidden), (kv, hidden), (hidden, q), (ffn, hidden), (ffn, hidden), (hidden, ffn)]
        size = sum(_weight_bytes(case["fmt"], n, k, 4) for n, k in shapes)
        size += 2 * m * (2 * hidden + q)                       # activations of the attention and feed-forward inputs
        size += 2 * m * (q + 2 * kv + 2 * hidden)              # q, k, v, o and down outputs
        if not fused:
            size += 2 * m * 3 * ffn                            # gate and up outputs, down's own input
        flops = sum(2 * m * n * k for n, k in shapes)
        return {"bytes": size * case["layers"], "flops": flops * case["layers"]}
    if kind == "linear":
        m, n, k = case["tokens"], case["n"], case["k"]
        return {"bytes": _weight_bytes(case["fmt"], n, k) + 2 * m * (k + n), "flops": 2 * m * n * k}
    if kind == "w8a8":
        m, shapes = case["tokens"], _layer_matrices(case)
        return {"bytes": sum(n * k + 2 * n + 2 * m * (k + n) for n, k in shapes),
                "flops": sum(2 * m * n * k for n, k in shapes)}
    if kind == "load":
        wide = 4 if case["dtype"] == "fp32" else 2
        return {"bytes": sum(wide * n * k + _weight_bytes(case["fmt"], n, k) for n, k in _layer_matrices(case)),
                "flops": 0}
    n, k = case["n"], case["k"]
    return {"bytes": _weight_bytes(case["fmt"], n, k) + 2 * n * k, "flops": 0}


def tolerance(case):
    """Relative 2-norm error another correct implementation may show: about four times what the path shows
    against the same products in 64 bits.  Measured there: one projection 2.1e-4 (int8) and 2.7e-4 (4-bit) in
    fp16, 1.7e-3 and 2.3e-3 in bf16; gate, up, SwiGLU and down in a row 4.2e-4 in fp16, 3.6e-3 in bf16."""
    kind = case["kind"]
    if kind in ("load", "dequant", "w8a8"):
        return "exact"        # bytes, and sums of integers: a pure function of the inputs
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 1.5e-3}
