"""The work this package does for its users, as measurable cases.

Weight-only quantised linears of the DreamZero / Wan transformer and of the layers around it,
called the way a model calls them: ``linear`` (the reference's ``ops.linear`` signature), the FFN
pair with its fused activation, one CUDA-graph replay of a stack of blocks, and the two ends of a
weight's life, ``quantize`` (load time) and ``dequantize`` (export, checks).

A case is a dict of plain values:

* ``op``      linear | ffn | blocks | quantize | dequantize
* ``m``       tokens (rows of the activations); ``batch`` > 0 gives them a leading dimension
* ``k``, ``n``  weight shape (input and output features; for ``ffn``: width and hidden width)
* ``bits``, ``group`` (0: one scale per output channel), ``symmetric``, ``bias``
"""
from __future__ import annotations

import math

import torch

import dexter_labs_b200 as d
from dexter_labs_b200 import ops, tp


def _case(op, m, k, n, bits=4, group=128, symmetric=False, bias=True, batch=0):
    return {"op": op, "m": m, "k": k, "n": n, "bits": bits, "group": group, "symmetric": symmetric,
            "bias": bias, "batch": batch}


def listed():
    def named(name, *args, **kwargs):
        return dict(_case(*args, **kwargs), name=name)

    return [
        # one token through an attention output projection of the 5B model: the smallest call,
        # asymmetric grid and bias as the model's own packing produces them
        named("o_w4_m1", "linear", 1, 3072, 3072),
        # a few tokens through the fused q/k/v projection
        named("qkv_w4_m8", "linear", 8, 3072, 9216),
        # the FFN of the 5B model at a control step's 83 tokens: up + tanh-GELU, then down
        named("ffn_w4_m83", "ffn", 83, 3072, 14336, symmetric=True),
        # the same with int8 weights, one scale per output channel
        named("ffn_w8_m83", "ffn", 83, 3072, 14336, bits=8, group=0, symmetric=True),
        # int8 in groups with zero points, activations with a leading batch dimension
        named("w8_b5_m125", "linear", 125, 3072, 8192, bits=8, batch=5),
        # the middle of the token range: two token blocks
        named("up_w4_m256", "linear", 256, 3072, 14336),
        # long K, few output tiles, int8 per channel
        named("down_w8_m512", "linear", 512, 14336, 3072, bits=8, group=0, symmetric=True),
        # the FFN of the 14B model at 913 tokens: the largest case, bound by the tensor cores
        named("ffn14b_w4_m913", "ffn", 913, 5120, 13824, symmetric=True),
        # a small layer outside the backbone: fine groups and an output width that is no
        # multiple of 16
        named("ragged_w4_m50", "linear", 50, 1536, 1000, group=32),
        # two whole blocks of the 5B model (twenty linears) as one captured graph, the
        # independent linears of a block side by side
        named("blocks5b_w4_m83", "blocks", 83, 3072, 14336, symmetric=True),
        # packing a weight when a model is loaded
        named("quantize_w4", "quantize", 0, 3072, 14336, bias=False),
        # the dense weight back from its packed form
        named("dequantize_w4", "dequantize", 0, 3072, 14336, bias=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["linear"] * 10 + ["ffn"] * 3 + ["blocks"] + ["quantize", "dequantize"] * 2)
    bits = rng.choice([4, 4, 8])
    group = 128 if bits == 4 else rng.choice([0, 128])
    symmetric, bias = rng.random() < 0.5, rng.random() < 0.75
    m = _log(rng, 1, 913)
    if op == "blocks":
        return _case(op, _log(rng, 1, 200), 3072, 14336, bits, group, symmetric, bias)
    if op in ("quantize", "dequantize"):
        # any output width: packing does not care about tiles
        return _case(op, 0, 256 * _log(rng, 1, 56), _log(rng, 64, 14336), bits, group, symmetric, False)
    if op == "ffn":
        k = 256 * _log(rng, 2, 20)
        return _case(op, m, k, 256 * _log(rng, k // 128, 54), bits, group, symmetric, bias)
    if rng.random() < 0.2:
        # small layers outside the backbone: fine groups, any output width
        group = rng.choice([32, 64, 128])
        return _case(op, _log(rng, 1, 128), 256 * rng.randint(1, 8), _log(rng, 33, 2048), bits, group,
                     symmetric, bias)
    k = 256 * _log(rng, 1, 56)
    n = 16 * _log(rng, 4, 896)
    batch = rng.choice([0, 0, 2])
    return _case(op, m + m % 2 if batch else m, k, n, bits, group, symmetric, bias, batch)


def _weight(case, k, n, gen):
    w = (torch.randn(n, k, generator=gen, device="cuda") * 0.02).to(torch.bfloat16)
    bias = None
    if case["bias"]:
        bias = (torch.randn(n, generator=gen, device="cuda") * 0.1).to(torch.bfloat16)
    return w, bias


def _packed(case, k, n, gen):
    w, bias = _weight(case, k, n, gen)
    return d.quantize(w, bits=case["bits"], group_size=case["group"] or k, bias=bias,
                      symmetric=case["symmetric"])


def _tokens(case, k, gen):
    x = torch.randn(case["m"], k, generator=gen, device="cuda").to(torch.bfloat16)
    return x.view(case["batch"], -1, k) if case["batch"] else x


_BLOCK = (("self_q", "column"), ("self_k", "column"), ("self_v", "column"), ("self_o", "row"),
          ("cross_q", "column"), ("cross_k", "column"), ("cross_v", "column"), ("cross_o", "row"),
          ("ffn_up", "column"), ("ffn_down", "row"))
_NUM_BLOCKS = 2


def _block_shape(case, name):
    k = case["n"] if name == "ffn_down" else case["k"]
    n = case["n"] if name == "ffn_up" else case["k"]
    return k, n


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op, k, n = case["op"], case["k"], case["n"]
    state = {"op": op, "bits": case["bits"], "group": case["group"] or k, "symmetric": case["symmetric"]}
    if op == "linear":
        state.update(w=_packed(case, k, n, gen), x=_tokens(case, k, gen))
    elif op == "ffn":
        state.update(up=_packed(case, k, n, gen), down=_packed(case, n, k, gen), x=_tokens(case, k, gen))
    elif op == "quantize":
        state.update(w=_weight(case, k, n, gen)[0])
    elif op == "dequantize":
        state.update(w=_packed(case, k, n, gen))
    else:
        layers = tp.LayerSet(dim=k, ffn_dim=n, blocks=_NUM_BLOCKS, bits=case["bits"],
                             group_size=case["group"], concurrent=True)
        for _ in range(_NUM_BLOCKS):
            layers.layers.append([layers.shard(name, kind, _packed(case, *_block_shape(case, name), gen))
                                  for name, kind in _BLOCK])
        layers.relayout_()
        x, ctx = _tokens(case, k, gen), _tokens(case, k, gen)
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            layers.forward(x, ctx)
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                y = layers.forward(x, ctx)
        torch.cuda.current_stream().wait_stream(stream)
        state.update(layers=layers, x=x, ctx=ctx, graph=graph, y=y)
    return state


def _linear(x, w):
    return d.linear(x, w.qweight, w.bias, scales=w.scales, zeros=w.zeros, group_size=w.group_size,
                    bits=w.bits)


def run(state):
    op = state["op"]
    if op == "linear":
        return _linear(state["x"], state["w"])
    if op == "ffn":
        up = state["up"]
        gelu = ops.w4a16_gelu if up.bits == 4 else ops.w8a16_gelu
        hidden = gelu(state["x"], up.qweight, up.scales, up.zeros, up.bias, up.group_size)
        return _linear(hidden, state["down"])
    if op == "quantize":
        q = d.quantize(state["w"], bits=state["bits"], group_size=state["group"],
                       symmetric=state["symmetric"])
        return {"qweight": q.qweight, "scales": q.scales, "zeros": q.zeros}
    if op == "dequantize":
        w = state["w"]
        return d.dequantize(w.qweight, w.scales, w.zeros, w.group_size, w.bits)
    state["graph"].replay()
    return state["y"]


def _weight_bytes(case, k, n):
    groups = k // (case["group"] or k)
    return k * n * case["bits"] // 8 + groups * n * 2 * (1 if case["symmetric"] else 2) + (2 * n if case["bias"] else 0)


def work(case):
    """Bytes of every input read once and every output written once, and the flops of the
    matrix products."""
    op, m, k, n = case["op"], case["m"], case["k"], case["n"]
    if op == "linear":
        return {"bytes": _weight_bytes(case, k, n) + 2 * m * (k + n), "flops": 2 * m * k * n}
    if op == "ffn":
        return {"bytes": _weight_bytes(case, k, n) + _weight_bytes(case, n, k) + 4 * m * k, "flops": 4 * m * k * n}
    if op in ("quantize", "dequantize"):
        return {"bytes": _weight_bytes(case, k, n) + 2 * k * n, "flops": 0}
    shapes = [_block_shape(case, name) for name, _ in _BLOCK] * _NUM_BLOCKS
    return {"bytes": sum(_weight_bytes(case, a, b) for a, b in shapes) + 6 * m * k,
            "flops": sum(2 * m * a * b for a, b in shapes)}


def tolerance(case):
    """Packing and unpacking are exact.  Products accumulate in fp32 and are rounded to bf16: another
    summation order moves a value by one bf16 step (2^-8) now and then, and by one more where a
    bias is added to the rounded product; a chain of linears carries that along."""
    if case["op"] in ("quantize", "dequantize"):
        return "exact"
    if case["op"] == "linear":
        return {"rel": 4e-3, "max": 0.02}
    if case["op"] == "ffn":
        return {"rel": 6e-3, "max": 0.03}
    return {"rel": 1e-2, "max": 0.06}
