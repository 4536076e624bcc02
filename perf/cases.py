"""What a user of this package has it do, as cases that can be timed: decode projections from one small eager call to
a 36-layer step, prompts from a short one to the 70B-class sweep, the decoder MLP, and dequantisation.

A case is a dict of plain values.  ``kind`` says which public entry point it goes through:

  call     ``tensor_b200.gguf(m, n, k, format)`` and ``launch(x, w, out)`` on the current stream; m <= 16 is a decode
           GEMV (bf16, fp16 or fp32 activations), a larger m a prefill GEMM (bf16)
  list     ``ShardedGemvList`` on one GPU: gate, up and down of one MLP at each of several batches, one call
  mlp      ``DecoderMlp``: norm, gate + up, SwiGLU, down, residual add
  step     the projections of all layers of a decoder for one token batch, each its own ``launch``, captured once in a
           CUDA graph and replayed per token (rows of q, k, v and of gate, up concatenated when the weights are loaded)
  dequant  ``tensor_b200.dequantize`` into an fp32 buffer the caller keeps
"""

from __future__ import annotations

import torch

import tensor_b200 as tb
from tensor_b200 import ops, synth
from tensor_b200.formats import get_format
from tensor_b200.projection import DecoderMlp, ShardedGemvList

DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}

# The largest prompt of the K-quants and of the plain 32-weight formats, and the largest single decode weight.
MAX_PROMPT = 4096 * 28672 * 8192
MAX_PROMPT_PLAIN = 333 * 12288 * 4096
MAX_WEIGHT = 28672 * 8192


def listed():
    return [
        # one k/v projection of a decoder with 8 key heads of 128: the smallest call, latency only
        {"name": "call_q4_k_1x1024x4096", "kind": "call", "format": "q4_k", "m": 1, "n": 1024, "k": 4096, "x": "bfloat16"},
        # a square attention projection kept in Q8_0, fp16 activations, one token
        {"name": "call_q8_0_1x4096x4096_f16", "kind": "call", "format": "q8_0", "m": 1, "n": 4096, "k": 4096, "x": "float16"},
        # an up projection in Q4_0 for eight sequences decoded together
        {"name": "call_q4_0_8x12288x4096", "kind": "call", "format": "q4_0", "m": 8, "n": 12288, "k": 4096, "x": "bfloat16"},
        # one MLP (18944 x 3584) in Q4_K serving batches of 1, 4 and 16 together: nine projections in one call
        {"name": "list_q4_k_18944x3584_b1_4_16", "kind": "list", "format": "q4_k", "batches": "1,4,16", "hidden": 3584,
         "inter": 18944},
        # the MLP block of a decoder layer with the mixed formats files are shipped with (down in Q6_K), four sequences
        {"name": "mlp_q4_k_q6_k_b4_4096x12288", "kind": "mlp", "format": "q4_k", "down": "q6_k", "m": 4, "hidden": 4096,
         "inter": 12288},
        # every projection of a 36-layer 8B-class decoder for one token, and for sixteen sequences
        {"name": "step_36x4096_b1", "kind": "step", "format": "q4_k", "down": "q6_k", "m": 1, "layers": 36, "hidden": 4096,
         "kv": 1024, "inter": 12288},
        {"name": "step_36x4096_b16", "kind": "step", "format": "q4_k", "down": "q6_k", "m": 16, "layers": 36, "hidden": 4096,
         "kv": 1024, "inter": 12288},
        # prompts: an ordinary one, a long one in the heavier format, and the 70B-class sweep
        {"name": "prompt_q4_k_512x12288x4096", "kind": "call", "format": "q4_k", "m": 512, "n": 12288, "k": 4096, "x": "bfloat16"},
        {"name": "prompt_q6_k_2048x12288x4096", "kind": "call", "format": "q6_k", "m": 2048, "n": 12288, "k": 4096, "x": "bfloat16"},
        {"name": "prompt_q4_k_4096x28672x8192", "kind": "call", "format": "q4_k", "m": 4096, "n": 28672, "k": 8192, "x": "bfloat16"},
        # a prompt of no round length through weights kept in Q8_0
        {"name": "prompt_q8_0_333x12288x4096", "kind": "call", "format": "q8_0", "m": 333, "n": 12288, "k": 4096, "x": "bfloat16"},
        # a weight expanded to fp32 (loading it into an unquantised layer)
        {"name": "dequant_q6_k_12288x4096", "kind": "dequant", "format": "q6_k", "n": 12288, "k": 4096},
    ]


def _log(rng, low, high):
    """An integer of [low, high], uniform in its logarithm."""
    return min(high, max(low, int(round(low * (high / low) ** rng.random()))))


def _rows(rng, low, high):
    """Rows of a weight: half of them a multiple of 128, the others whatever a vocabulary or a slice leaves."""
    n = _log(rng, low, high)
    return max(128, n // 128 * 128) if rng.random() < 0.5 else n


def _inner(rng, fmt, low, high):
    step = get_format(fmt).weights
    return step * _log(rng, -(-low // step), high // step)


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "prompt", "mlp", "step", "list", "dequant"])
    fmt = rng.choice(["q4_k", "q4_k", "q6_k", "q8_0", "q4_0"])
    if kind == "decode":
        m = 1 if rng.random() < 0.5 else rng.randint(2, 16)
        x = rng.choice(["bfloat16"] * 6 + ["float16"] * 3 + ["float32"])
        while True:
            n, k = _rows(rng, 256, 32768), _inner(rng, fmt, 512, 28672)
            if n * k <= MAX_WEIGHT:
                return {"kind": "call", "format": fmt, "m": m, "n": n, "k": k, "x": x}
    if kind == "prompt":
        most = MAX_PROMPT if fmt in ("q4_k", "q6_k") else MAX_PROMPT_PLAIN
        while True:
            m, n, k = _log(rng, 17, 4096), _rows(rng, 256, 28672), _inner(rng, fmt, 512, 28672)
            if n * k <= MAX_WEIGHT and m * n * k <= most:
                return {"kind": "call", "format": fmt, "m": m, "n": n, "k": k, "x": "bfloat16"}
    if kind == "dequant":
        while True:
            n, k = _rows(rng, 256, 32768), _inner(rng, fmt, 512, 28672)
            if n * k <= MAX_WEIGHT:
                return {"kind": "dequant", "format": fmt, "n": n, "k": k}
    hidden = 256 * rng.randint(8, 24)  # decoders' widths: multiples of 256 in every format here
    inter = 256 * _log(rng, hidden // 128, hidden // 64 + hidden // 512)
    m = 1 if rng.random() < 0.4 else rng.randint(2, 16)
    if kind == "mlp":
        return {"kind": "mlp", "format": fmt, "down": rng.choice([fmt, "q6_k"]), "m": m, "hidden": hidden, "inter": inter}
    if kind == "list":
        return {"kind": "list", "format": fmt, "batches": rng.choice(["1", "1,4,16", "%d" % m, "1,%d" % rng.randint(2, 16)]),
                "hidden": hidden, "inter": inter}
    return {"kind": "step", "format": fmt, "down": rng.choice([fmt, "q6_k"]), "m": m, "layers": _log(rng, 2, 24),
            "hidden": hidden, "kv": hidden // rng.choice([1, 4]), "inter": min(inter, 3 * hidden)}


def _projections(case):
    """(format, rows, K, activation group) of the four launches of a decoder layer."""
    h, kv, i = case["hidden"], case["kv"], case["inter"]
    return [(case["format"], h + 2 * kv, h, 0), (case["format"], h, h, 1), (case["format"], 2 * i, h, 2), (case["down"], h, i, 3)]


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    seed = seed * 1009 + 17
    kind = case["kind"]
    if kind == "call":
        m, n, k, fmt = case["m"], case["n"], case["k"], case["format"]
        return {"kind": kind, "kernel": tb.gguf(m, n, k, fmt, x_dtype=case["x"]),
                "x": synth.make_activations(m, k, seed, dev, DTYPES[case["x"]]),
                "w": synth.make_weights(fmt, n, k, seed + 1, dev),
                "out": torch.empty((m, n), dtype=torch.float32, device=dev)}
    if kind == "dequant":
        n, k = case["n"], case["k"]
        return {"kind": kind, "format": case["format"], "n": n, "k": k, "w": synth.make_weights(case["format"], n, k, seed, dev),
                "out": torch.empty((n, k), dtype=torch.float32, device=dev)}
    if kind == "mlp":
        m, h, i = case["m"], case["hidden"], case["inter"]
        gen = torch.Generator(device=dev)
        gen.manual_seed(seed)
        block = DecoderMlp(synth.make_weights(case["format"], i, h, seed + 1, dev), synth.make_weights(case["format"], i, h, seed + 2, dev),
                           synth.make_weights(case["down"], h, i, seed + 3, dev),
                           1 + 0.1 * torch.randn(h, generator=gen, device=dev), h, i, m, case["format"], case["down"])
        return {"kind": kind, "block": block, "h": torch.randn((m, h), generator=gen, device=dev)}
    if kind == "list":
        h, i, fmt = case["hidden"], case["inter"], case["format"]
        gate, up, down = (synth.make_weights(fmt, n, k, seed + j, dev) for j, (n, k) in enumerate([(i, h), (i, h), (h, i)]))
        specs = []
        for b in (int(v) for v in case["batches"].split(",")):
            x, act = synth.make_activations(b, h, seed + 10 + b, dev), synth.make_activations(b, i, seed + 40 + b, dev)
            specs += [(x, gate, fmt, i, h), (x, up, fmt, i, h), (act, down, fmt, h, i)]
        return {"kind": kind, "list": ShardedGemvList(specs)}
    # a whole decode step: one kernel per shape, the weights of every layer, one graph replayed per token
    m, parts = case["m"], _projections(case)
    weights = [[synth.make_weights(fmt, n, k, seed + 8 * layer + j, dev) for j, (fmt, n, k, _) in enumerate(parts)]
               for layer in range(case["layers"])]
    xs = [synth.make_activations(m, k, seed + 1000 + g, dev) for _, _, k, g in parts]
    outs = [torch.empty((case["layers"], m, n), dtype=torch.float32, device=dev) for _, n, _, _ in parts]
    kernels = [tb.gguf(m, n, k, fmt, device=dev) for fmt, n, k, _ in parts]

    def step():
        for layer in range(case["layers"]):
            for j, kernel in enumerate(kernels):
                kernel.launch(xs[j], weights[layer][j], outs[j][layer])

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    return {"kind": kind, "graph": graph, "outs": outs, "keep": (weights, xs, kernels)}


def run(state):
    kind = state["kind"]
    if kind == "call":
        return state["kernel"].launch(state["x"], state["w"], state["out"])
    if kind == "list":
        return state["list"].forward()
    if kind == "mlp":
        return state["block"].forward(state["h"])
    if kind == "step":
        state["graph"].replay()
        return state["outs"]
    return ops.dequantize(state["w"], state["format"], state["n"], state["k"], out=state["out"])


def _gemm_work(fmt, m, n, k, x_bytes=2, weights=True):
    moved = (get_format(fmt).weight_bytes(n, k) if weights else 0) + m * k * x_bytes + m * n * 4
    return moved, 2.0 * m * n * k


def work(case):
    kind = case["kind"]
    if kind == "dequant":
        n, k = case["n"], case["k"]
        return {"bytes": get_format(case["format"]).weight_bytes(n, k) + 4 * n * k, "flops": 1.0 * n * k}
    if kind == "call":
        parts = [_gemm_work(case["format"], case["m"], case["n"], case["k"], 4 if case["x"] == "float32" else 2)]
    elif kind == "step":
        parts = [_gemm_work(fmt, case["m"], n, k) for fmt, n, k, _ in _projections(case)] * case["layers"]
    else:
        h, i, fmt = case["hidden"], case["inter"], case["format"]
        batches = [case["m"]] if kind == "mlp" else [int(v) for v in case["batches"].split(",")]
        # a list reads each of its three weights once for all its batches
        parts = [_gemm_work(f, b, n, k, weights=b == batches[0])
                 for b in batches for f, n, k in [(fmt, i, h), (fmt, i, h), (case.get("down", fmt), h, i)]]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    if case["kind"] == "dequant":
        return "exact"  # the decode is one correctly rounded operation after another
    if case["kind"] == "mlp":
        return {"rel": 4e-3}  # two activations rounded to bf16 on the way (2^-9 each)
    # products of the same operands (exact for a GEMV, bf16 for a GEMM), summed in fp32 in some order over up to 28672 terms
    return {"rel": 2e-5}
