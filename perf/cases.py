"""Timed workloads of the W4A16 path, through the package's public entry points.

Three kinds of pass:

* ``linear`` - ``BlkQ4Linear.forward`` on ``layers`` layers of one shape, each with its own weights and
  all reading the same activation, called one after the other as an eager model calls them;
* ``stack``  - ``LinearStack.forward``: the seven linears of ``blocks`` decoder blocks, replayed as one
  CUDA graph (``llama_like_stack``);
* ``quant``  - ``ms_blkq4linear_ext.quant`` on a list of fp16 weight matrices: what constructing layers
  from an fp16 checkpoint does.

Weights are N(0, 0.02), activations N(0, 1), as the benchmark and the tests have them.
"""
from __future__ import annotations

import math

import torch

from gemmlib_b200 import ms_blkq4linear_ext
from gemmlib_b200.ms_blkq4linear import BlkQ4Linear
from gemmlib_b200.stack import llama_like_stack

SIGMA = 0.02


def _linear(name, m, k, n, block, col_wise, zp, bias, layers):
    return dict(name=name, kind="linear", m=m, k=k, n=n, block=block, col_wise=col_wise, zp=zp, bias=bias,
                layers=layers)


def _stack(name, m, hidden, ffn, blocks, block, col_wise, zp):
    return dict(name=name, kind="stack", m=m, hidden=hidden, ffn=ffn, blocks=blocks, block=block,
                col_wise=col_wise, zp=zp)


def _quant(name, what, k, n, block, col_wise, zp):
    return dict(name=name, kind="quant", what=what, k=k, n=n, block=block, col_wise=col_wise, zp=zp)


def listed():
    return [
        # One token through one attention projection, called on its own: launch and host latency.
        _linear("linear_m1_4096", 1, 4096, 4096, 64, True, True, False, 1),
        # One token through the up projections of sixteen blocks, eager: 384 MB of weights, more than L2.
        _linear("linear_m1_11008_x16", 1, 4096, 11008, 64, True, False, False, 16),
        # Decode step of two decoder blocks as one CUDA graph (222 MB of weights).
        _stack("stack_m1", 1, 4096, 11008, 2, 64, True, True),
        # Four sequences through a large MLP projection with bias.
        _linear("linear_m4_28672", 4, 8192, 28672, 128, True, False, True, 1),
        # A batch of sixteen on small blocks with zero points; four layers.
        _linear("linear_m16_b32_x4", 16, 4096, 4096, 32, True, True, False, 4),
        # A batch of 64 sequences on the large projection: between memory and tensor bound.
        _linear("linear_m64_28672", 64, 8192, 28672, 128, True, False, False, 1),
        # Row-wise blocks, ragged in every direction, with bias.
        _linear("linear_rowwise_m333", 333, 4032, 2080, 32, False, True, True, 1),
        # A prompt of 512 tokens through one decoder block as one CUDA graph.
        _stack("stack_m512", 512, 4096, 11008, 1, 64, True, True),
        # A long prompt through an attention projection, small blocks with zero points.
        _linear("linear_m2048_b32", 2048, 4096, 4096, 32, True, True, False, 1),
        # The largest: 4096 tokens through the large projection.
        _linear("linear_m4096_28672", 4096, 8192, 28672, 128, True, False, False, 1),
        # Quantize and prepack the seven weights of a decoder block.
        _quant("quant_block", "block", 4096, 11008, 64, True, True),
        # Quantize and prepack one weight with row-wise blocks, symmetric.
        _quant("quant_rowwise", "one", 11008, 4096, 32, False, False),
    ]


def _log_size(rng, lo, hi, multiple):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // multiple, max(-(-lo // multiple), round(v / multiple))) * multiple


def draw(rng):
    kind = rng.choice(["linear"] * 6 + ["stack"] * 2 + ["quant"] * 2)
    block = rng.choice([16, 32, 32, 64, 64, 64, 128, 128])
    col_wise = rng.random() < 0.8
    zp = rng.random() < 0.5
    k_mult = max(64, block) if col_wise else 64
    n_mult = 32 if col_wise else max(32, block)
    if kind == "stack":
        hidden = _log_size(rng, 1024, 4096, 128)
        ffn = _log_size(rng, hidden, 11008, 128)
        c = _stack("", _log_size(rng, 1, 512, 1), hidden, ffn, rng.choice([1, 2]), block, col_wise, zp)
    elif kind == "quant":
        what = rng.choice(["one", "one", "block"])
        if what == "block":
            k = _log_size(rng, 1024, 4096, 128)
            n = _log_size(rng, k, 11008, 128)
        else:
            k, n = _log_size(rng, 512, 11008, k_mult), _log_size(rng, 512, 28672, n_mult)
        c = _quant("", what, k, n, block, col_wise, zp)
    else:
        m = _log_size(rng, 1, 4096, 1)
        k, n = _log_size(rng, 512, 11008, k_mult), _log_size(rng, 512, 28672, n_mult)
        c = _linear("", m, k, n, block, col_wise, zp, rng.random() < 0.4, rng.choice([1, 1, 2, 4]) if m <= 64 else 1)
    del c["name"]
    return c


def _block_shapes(hidden, ffn):
    """(out_features, in_features) of the seven linears of a decoder block."""
    return [(hidden, hidden)] * 4 + [(ffn, hidden)] * 2 + [(hidden, ffn)]


def _quant_shapes(case):
    return _block_shapes(case["k"], case["n"]) if case["what"] == "block" else [(case["n"], case["k"])]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(rows, cols, sigma):
        return torch.randn(rows, cols, generator=gen, device="cuda", dtype=torch.float32).mul_(sigma).to(torch.float16)

    kind, block, col_wise, zp = case["kind"], case["block"], case["col_wise"], case["zp"]
    if kind == "quant":
        return dict(kind=kind, block=block, col_wise=col_wise, zp=zp,
                    weights=[normal(n, k, SIGMA) for n, k in _quant_shapes(case)])
    if kind == "stack":
        stack = llama_like_stack(case["hidden"], case["ffn"], case["blocks"], block, col_wise, not zp,
                                 torch.device("cuda"), weight_fn=lambda n, k: normal(n, k, SIGMA))
        stack.buffers(case["m"])  # the graph of this row count is captured once and kept
        return dict(kind=kind, stack=stack, m=case["m"], x=normal(case["m"], case["hidden"], 1.0),
                    result=f"h{(case['blocks'] - 1) % 2}")
    layers = []
    for _ in range(case["layers"]):
        bias = normal(1, case["n"], SIGMA).view(-1) if case["bias"] else None
        layers.append(BlkQ4Linear(block, col_wise, not zp, normal(case["n"], case["k"], SIGMA), bias))
    return dict(kind=kind, layers=layers, x=normal(case["m"], case["k"], 1.0))


def run(state):
    if state["kind"] == "linear":
        x = state["x"]
        return [layer(x) for layer in state["layers"]]
    if state["kind"] == "stack":
        stack = state["stack"]
        hidden = stack.forward(state["x"], state["result"])
        return dict(stack.buffers(state["m"]), result=hidden)
    return [ms_blkq4linear_ext.quant(state["block"], state["col_wise"], state["zp"], w) for w in state["weights"]]


def _packed_bytes(n, k, block, zp):
    meta = n * k // block
    return n * k // 2 + 2 * meta + (meta if zp else 0)


def work(case):
    block, zp = case["block"], case["zp"]
    if case["kind"] == "quant":
        return {"bytes": sum(2 * n * k + _packed_bytes(n, k, block, zp) for n, k in _quant_shapes(case)), "flops": 0}
    m = case["m"]
    if case["kind"] == "stack":
        shapes = _block_shapes(case["hidden"], case["ffn"]) * case["blocks"]
        once = 2 * m * case["hidden"]
    else:
        shapes = [(case["n"], case["k"])] * case["layers"]
        once = 2 * m * case["k"] + (2 * case["n"] * case["layers"] if case["bias"] else 0)
    return {"bytes": once + sum(_packed_bytes(n, k, block, zp) + 2 * m * n for n, k in shapes),
            "flops": sum(2 * m * n * k for n, k in shapes)}


def tolerance(case):
    """The quantizer's bytes are fixed by the format.  A linear's result is rounded to fp16 (2^-11) and its
    weights may be dequantized with up to two fp16 roundings of terms up to 31 scales, half a unit of
    which is 0.4 % of a scale, on weights of a few scales; in the stack four to eight linears follow one another."""
    if case["kind"] == "quant":
        return "exact"
    return {"rel": 1e-2 if case["kind"] == "stack" else 4e-3}
