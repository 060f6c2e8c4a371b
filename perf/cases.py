"""Performance cases of the quantized linear path, through the public entry points (`ops.Context`, `ops.Linear`).

The sizes are those of the benchmark's synthetic decoder (hidden 2048, fused QKV 4096, fused gate+up 12288, down
6144 -> 2048, 28 layers, up to 64 decode streams, prefill of thousands of tokens) and of the encoder-side blocks the
row-wise operators are tested with (widths 256 to 2048, LayerNorm, bias, activation, residual). Values follow the
benchmark's distributions: N(0,1) activations with a few outlier channels (heavy-tailed Student-t for the K-group
modes), N(0, 0.02) weights.

Kinds of case:
  linear   one `Linear.forward` called eagerly: a dense activation is quantized, multiplied, finished. What a program
           pays per projection when it does not capture its step; a few rows, so latency and host work count.
  decode   one step of the 28-layer stack for `rows` concurrent streams, captured once as a CUDA graph and replayed,
           as a serving loop does.
  prefill  one decoder layer over a prompt (or a batch of prompts) of `rows` tokens, called eagerly; prompts have any
           length, so the row counts are ragged.
  block    LayerNorm -> up projection (bias, activation) -> down projection (bias, residual), the feed-forward half of
           an encoder or a diffusion block; `modulated` adds the per-sequence shift, scale and gate of the latter.
  load     quantization of one weight matrix when a model is loaded.
"""
import math

import torch

from breeze_tts_cpp_b200 import ops

HIDDEN, QKV, FFN, LAYERS = 2048, 4096, 6144, 28
PROJECTIONS = {"qkv": (HIDDEN, QKV), "o": (HIDDEN, HIDDEN), "gate_up": (HIDDEN, 2 * FFN), "down": (FFN, HIDDEN)}  # K, N
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}
ACTIVATIONS = {"relu": ops.RELU, "gelu": ops.GELU, "gelu_tanh": ops.GELU_TANH, "silu": ops.SILU}
EPSILON = 1e-6


def listed():
    return [
        # One stream, one small projection, nothing captured: the smallest call there is.
        {"name": "linear_o_int8_m1", "kind": "linear", "mode": "int8", "projection": "o", "rows": 1, "dtype": "bf16",
         "bias": False, "residual": False},
        # A batch of streams through the K-group down projection with its residual.
        {"name": "linear_down_group_int8_m16", "kind": "linear", "mode": "group_int8", "projection": "down", "rows": 16,
         "dtype": "bf16", "bias": False, "residual": True},
        # A full machine of decode streams: the benchmark's own workload.
        {"name": "decode_int8_m64", "kind": "decode", "mode": "int8", "rows": 64},
        # A few interactive streams.
        {"name": "decode_fp8_m5", "kind": "decode", "mode": "fp8", "rows": 5},
        # One prompt of ordinary, ragged length.
        {"name": "prefill_int8_m301", "kind": "prefill", "mode": "int8", "rows": 301},
        # Some long prompts in the K-group mode, ragged.
        {"name": "prefill_group_fp8_m1021", "kind": "prefill", "mode": "group_fp8", "rows": 1021},
        # The benchmark's prefill sizes.
        {"name": "prefill_fp8_m2048", "kind": "prefill", "mode": "fp8", "rows": 2048},
        {"name": "prefill_group_int8_m4096", "kind": "prefill", "mode": "group_int8", "rows": 4096},
        {"name": "prefill_int8_m8192", "kind": "prefill", "mode": "int8", "rows": 8192},
        # Encoder feed-forward block over some seconds of frames.
        {"name": "block_int8_w1024_m750", "kind": "block", "mode": "int8", "dtype": "f16", "sequences": 1, "length": 750,
         "width": 1024, "activation": "gelu", "modulated": False},
        # Narrow diffusion block over a batch of sequences.
        {"name": "block_fp8_w512_m4x93", "kind": "block", "mode": "fp8", "dtype": "bf16", "sequences": 4, "length": 93,
         "width": 512, "activation": "relu", "modulated": True},
        # Loading the largest matrix of a layer in the K-group mode.
        {"name": "load_group_int8_gate_up", "kind": "load", "mode": "group_int8", "channels": 2 * FFN, "reduction": HIDDEN,
         "dtype": "bf16"},
    ]


def _spread(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(["linear"] * 3 + ["decode"] * 2 + ["prefill"] * 4 + ["block"] * 3 + ["load"])
    mode = rng.choice(ops.MODES)
    if kind == "linear":
        return {"kind": kind, "mode": mode, "projection": rng.choice(sorted(PROJECTIONS)), "rows": _spread(rng, 1, 64),
                "dtype": rng.choice(sorted(DTYPES)), "bias": rng.random() < 0.5, "residual": rng.random() < 0.5}
    if kind == "decode":
        return {"kind": kind, "mode": mode, "rows": _spread(rng, 1, 64)}
    if kind == "prefill":
        return {"kind": kind, "mode": mode, "rows": _spread(rng, 65, 4096 if mode.startswith("group") else 8192)}
    if kind == "block":
        sequences = rng.choice((1, 2, 4, 8))
        return {"kind": kind, "mode": mode, "dtype": rng.choice(sorted(DTYPES)), "sequences": sequences,
                "length": _spread(rng, 16, 4096 // sequences), "width": rng.choice((256, 384, 512, 768, 1024, 1536, 2048)),
                "activation": rng.choice(sorted(ACTIVATIONS)), "modulated": rng.random() < 0.4}
    return {"kind": kind, "mode": mode, "channels": 16 * _spread(rng, 64, 768), "reduction": 128 * _spread(rng, 4, 48),
            "dtype": rng.choice(sorted(DTYPES))}


# ---------------------------------------------------------------------------------------------------------- inputs
class _Source:
    """Seeded tensors on the GPU, one generator for all of a state."""

    def __init__(self, seed):
        self.generator = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, rows, cols, std=1.0, mean=0.0, dtype=torch.bfloat16):
        return (torch.randn(rows, cols, generator=self.generator, device="cuda") * std + mean).to(dtype)

    def weight(self, rows, cols, dtype=torch.bfloat16):
        return torch.randn(rows, cols, generator=self.generator, device="cuda", dtype=dtype).mul_(0.02)

    def activation(self, rows, cols, mode, dtype=torch.bfloat16):
        x = torch.randn(rows, cols, generator=self.generator, device="cuda")
        if mode.startswith("group"):  # Student-t, 3 degrees of freedom
            chi2 = torch.zeros_like(x)
            for _ in range(3):
                chi2 += torch.randn(rows, cols, generator=self.generator, device="cuda").square_()
            x = x / (chi2 / 3).sqrt().clamp_min(1e-2)
        else:
            x[:, torch.randperm(cols, generator=self.generator, device="cuda")[:max(1, round(cols * 0.005))]] *= 20.0
        return x.to(dtype)


def _quantized(ctx, mode, matrix):
    group, _, rotation = ops.groups_of(mode)
    view = ops.RowScaledView.empty(matrix.shape[0], matrix.shape[1], ops.format_of(mode), group, rotation)
    return ctx.quantize_rows(matrix, view)


class _Layer:
    """Quantized weights and norm weights of one decoder layer."""

    def __init__(self, ctx, mode, rows, source):
        for name, (k, n) in PROJECTIONS.items():
            weight = _quantized(ctx, mode, source.weight(n, k))
            ctx.prepare_quantized(rows, n, k, weight=weight)
            setattr(self, name, weight)
        self.pre, self.post = (source.normal(1, HIDDEN, 0.1, 1.0) for _ in range(2))


class _Buffers:
    """The activation buffers a decoder keeps for `rows` tokens."""

    def __init__(self, mode, rows, source):
        group, _, rotation = ops.groups_of(mode)
        self.x0 = source.activation(rows, HIDDEN, mode)
        self.x = self.x0.clone()
        self.qkv = torch.empty(rows, QKV, dtype=torch.bfloat16, device="cuda")
        self.u = torch.zeros(rows, HIDDEN, dtype=torch.bfloat16, device="cuda")
        self.gate_up = torch.empty(rows, 2 * FFN, dtype=torch.bfloat16, device="cuda")
        self.q_hidden = ops.RowScaledView.empty(rows, HIDDEN, ops.format_of(mode), group, rotation)
        self.q_ffn = ops.RowScaledView.empty(rows, FFN, ops.format_of(mode), group, rotation)


def _decoder_layer(ctx, layer, b, update):
    ctx.quantized_norm(b.x, update, layer.pre, b.q_hidden, EPSILON)
    ctx.matmul(b.q_hidden, layer.qkv, b.qkv)
    ctx.quantize_rows(b.qkv[:, :HIDDEN], b.q_hidden)  # stands for the attention output, another subsystem's
    ctx.matmul(b.q_hidden, layer.o, b.u)
    ctx.quantized_norm(b.x, b.u, layer.post, b.q_hidden, EPSILON)
    ctx.matmul(b.q_hidden, layer.gate_up, b.gate_up)
    ctx.quantized_gated(b.gate_up, b.q_ffn)
    ctx.matmul(b.q_ffn, layer.down, b.u)


# --------------------------------------------------------------------------------------------------------- prepare
class _State:
    pass


def _prepare_linear(case, source, s):
    dtype, (k, n), rows = DTYPES[case["dtype"]], PROJECTIONS[case["projection"]], case["rows"]
    s.ctx = ops.Context(case["mode"])
    bias = source.normal(1, n, 0.3, dtype=dtype) if case["bias"] else None
    s.layer = ops.Linear(s.ctx, [source.weight(n, k, dtype)], bias=bias, max_rows=rows)
    s.x = source.activation(rows, k, case["mode"], dtype)
    s.out = torch.empty(rows, n, dtype=dtype, device="cuda")
    s.epilogue = {"residual": source.normal(rows, n, dtype=dtype)} if case["residual"] else {}


_capture_stream = None


def _prepare_decode(case, source, s):
    global _capture_stream
    if _capture_stream is None:
        _capture_stream = torch.cuda.Stream()
    _capture_stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(_capture_stream):
        s.ctx = ops.Context(case["mode"], stream=_capture_stream)
        s.layers = [_Layer(s.ctx, case["mode"], case["rows"], source) for _ in range(LAYERS)]
        s.buffers = _Buffers(case["mode"], case["rows"], source)
        s.ctx.seal()
        _decoder_layer(s.ctx, s.layers[0], s.buffers, None)  # loads the kernels before the capture
        _capture_stream.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph, stream=_capture_stream):
            s.buffers.x.copy_(s.buffers.x0, non_blocking=True)  # this step's tokens enter the residual stream
            for index, layer in enumerate(s.layers):
                _decoder_layer(s.ctx, layer, s.buffers, s.buffers.u if index else None)
    torch.cuda.current_stream().wait_stream(_capture_stream)


def _prepare_prefill(case, source, s):
    s.ctx = ops.Context(case["mode"])
    s.layer = _Layer(s.ctx, case["mode"], case["rows"], source)
    s.buffers = _Buffers(case["mode"], case["rows"], source)
    s.branch = source.normal(case["rows"], HIDDEN)  # what the layer before left to be added to the residual stream


def _prepare_block(case, source, s):
    dtype, width, rows = DTYPES[case["dtype"]], case["width"], case["sequences"] * case["length"]
    inner = 4 * width
    s.ctx = ops.Context(case["mode"])
    s.up = ops.Linear(s.ctx, [source.weight(inner, width, dtype)], bias=source.normal(1, inner, 0.3, dtype=dtype), max_rows=rows)
    s.down = ops.Linear(s.ctx, [source.weight(width, inner, dtype)], bias=source.normal(1, width, 0.3, dtype=dtype), max_rows=rows)
    s.x = source.activation(rows, width, case["mode"], dtype)
    s.gamma, s.beta = source.normal(1, width, 0.1, 1.0, dtype), source.normal(1, width, 0.1, dtype=dtype)
    s.h, s.y = torch.empty(rows, inner, dtype=dtype, device="cuda"), torch.empty(rows, width, dtype=dtype, device="cuda")
    s.fusion, s.epilogue = None, {"residual": s.x}
    s.activation = ACTIVATIONS[case["activation"]]
    if case["modulated"]:
        shift, scale, gate = (source.normal(case["sequences"], width, 0.2, dtype=dtype) for _ in range(3))
        s.fusion = {"shift": shift, "scale": scale, "rows_per_sequence": case["length"]}
        s.epilogue.update(gate=gate, rows_per_sequence=case["length"])


def _prepare_load(case, source, s):
    s.ctx = ops.Context(case["mode"])
    s.weight = source.weight(case["channels"], case["reduction"], DTYPES[case["dtype"]])
    group, _, rotation = ops.groups_of(case["mode"])
    s.view = ops.RowScaledView.empty(case["channels"], case["reduction"], ops.format_of(case["mode"]), group, rotation)


_PREPARE = {"linear": _prepare_linear, "decode": _prepare_decode, "prefill": _prepare_prefill, "block": _prepare_block,
            "load": _prepare_load}


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    _PREPARE[s.kind](case, _Source(seed), s)
    return s


# ------------------------------------------------------------------------------------------------------------- run
def run(s):
    if s.kind == "linear":
        return s.layer.forward(s.x, s.out, **s.epilogue)
    if s.kind == "decode":
        s.graph.replay()
        return {"residual": s.buffers.x, "branch": s.buffers.u}
    if s.kind == "prefill":
        b = s.buffers
        b.x.copy_(b.x0)  # the residual stream as the layer before left it; the layer updates it in place
        _decoder_layer(s.ctx, s.layer, b, s.branch)
        return {"qkv": b.qkv, "residual": b.x, "branch": b.u}
    if s.kind == "block":
        s.up.normalized_forward(s.x, s.h, s.gamma, s.beta, 1e-5, fusion=s.fusion, activation=s.activation)
        return s.down.forward(s.h, s.y, **s.epilogue)
    s.ctx.quantize_rows(s.weight, s.view)
    return {"values": s.view.values, "scales": s.view.scales}


# ---------------------------------------------------------------------------------------------------- work, tolerance
def _weight_bytes(mode, n, k):
    return n * k + 4 * n * (k // 128 if mode.startswith("group") else 1)


def work(case):
    kind, mode = case["kind"], case["mode"]
    if kind == "linear":
        (k, n), m = PROJECTIONS[case["projection"]], case["rows"]
        extra = (2 * n if case["bias"] else 0) + (2 * m * n if case["residual"] else 0)
        return {"bytes": 2 * m * k + _weight_bytes(mode, n, k) + 2 * m * n + extra, "flops": 2 * m * n * k}
    if kind in ("decode", "prefill"):
        m, layers = case["rows"], LAYERS if kind == "decode" else 1
        weights = sum(_weight_bytes(mode, n, k) for k, n in PROJECTIONS.values()) + 4 * HIDDEN
        # decode: the step's tokens in, residual and branch out; prefill: residual and branch in, both and QKV out
        rows = 3 * 2 * m * HIDDEN if kind == "decode" else 4 * 2 * m * HIDDEN + 2 * m * QKV
        return {"bytes": layers * weights + rows, "flops": layers * sum(2 * m * n * k for k, n in PROJECTIONS.values())}
    if kind == "block":
        m, w = case["sequences"] * case["length"], case["width"]
        modulation = 3 * 2 * case["sequences"] * w if case["modulated"] else 0
        return {"bytes": _weight_bytes(mode, 4 * w, w) + _weight_bytes(mode, w, 4 * w) + 2 * 7 * w + 2 * 2 * m * w + modulation,
                "flops": 2 * 2 * m * w * 4 * w}
    n, k = case["channels"], case["reduction"]
    return {"bytes": 2 * n * k + _weight_bytes(mode, n, k), "flops": 3 * n * k}


def tolerance(case):
    if case["kind"] == "load":
        return "exact"  # one-byte values and their scales are defined to the bit
    if case["kind"] == "decode":
        return {"rel": 2e-2}  # 28 layers of 16-bit rounding and 8-bit requantization in a row
    return {"rel": 1e-2 if case.get("dtype", "bf16") == "bf16" else 5e-3}  # 16-bit outputs of 8-bit operands
