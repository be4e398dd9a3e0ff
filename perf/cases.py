"""What this framework is asked to do, as cases that can be timed: ``listed()`` and ``draw()`` give them,
``prepare()`` makes what a program has in hand before the call, ``run()`` is one pass through the public
entry points, ``work()`` what the pass cannot do without and ``tolerance()`` how far two correct
implementations may be apart.

Five kinds of work, by ``op``:

* ``linear``  one quantised linear layer, ``DecodeLinear(x)``: fp16 activations, fp32 result.  Few rows are a
  decoding step, some tens a batch of requests, hundreds and more the prompt of a request (prefill).
* ``stack``   one pass of a [batch, hidden] residual stream through the linear layers of a transformer,
  ``LinearStack.step``: what a token costs.
* ``int8``    the integer operator, ``decode_matmul_cuda.decode_matmul(x, codes, codebook)``: a new int32 result.
* ``int8_inplace``  ``fast_decode_matmul_cuda.decode_matmul(x, codes, codebook, output)``: its own code layout
  and sign convention, added to the output.
* ``weights`` the decoded fp16 matrix itself, ``decode_weights``: export, inspection, another library's GEMM.
"""
import math

import torch

import decode_matmul_b200 as dmm
from decode_matmul_b200.linear import LLAMA2_70B, LLAMA2_7B, DecodeLinear, LinearStack, llama_shapes
from decode_matmul_cuda import decode_matmul as decode_matmul_int8
from fast_decode_matmul_cuda import decode_matmul as decode_matmul_int8_inplace

SCALE = 2.0 ** -12  # of a weight unit: keeps the residual stream of 80 blocks of random weights in range


def _stack(name, cfg, batch, **kw):
    return dict({"name": name, "op": "stack", "batch": batch, "codebook": "synthetic"}, **dict(cfg, **kw))


def listed():
    return [
        # the integer operator at the size its own test script calls it with: nothing but latency
        dict(name="int8_8x16x4096", op="int8", batch=8, n=16, k=4096, codebook="e8p"),
        # a Llama-2-7B q/k/v/o projection for one token: a small call on its own
        dict(name="linear_1x4096x4096", op="linear", batch=1, n=4096, k=4096, codebook="synthetic"),
        # a token of Llama-2-7B: 32 blocks of four products, four requests at a time
        _stack("stack_7b_b4", LLAMA2_7B, 4),
        # the decoding step that the benchmark reports: all 80 blocks of Llama-2-70B for one token ...
        _stack("stack_70b_b1", LLAMA2_70B, 1),
        # ... and for sixteen requests at a time
        _stack("stack_70b_b16", LLAMA2_70B, 16),
        # a batch of requests on the 70B gate (or up) projection
        dict(name="linear_32x28672x8192", op="linear", batch=32, n=28672, k=8192, codebook="synthetic"),
        # the largest batch of the 7B sweep, on the down projection
        dict(name="linear_64x4096x11008", op="linear", batch=64, n=4096, k=11008, codebook="e8p"),
        # a short prompt of no round length through a 7B gate projection
        dict(name="linear_333x11008x4096", op="linear", batch=333, n=11008, k=4096, codebook="e8p"),
        # a long prompt through the 70B down projection: the largest call
        dict(name="linear_2048x8192x28672", op="linear", batch=2048, n=8192, k=28672, codebook="synthetic"),
        # the integer operator at its usual eight rows on a 70B projection
        dict(name="int8_8x28672x8192", op="int8", batch=8, n=28672, k=8192, codebook="e8p"),
        # the in-place integer operator, a ragged batch
        dict(name="int8_inplace_13x8192x8192", op="int8_inplace", batch=13, n=8192, k=8192, codebook="e8p"),
        # export of one 7B projection to fp16
        dict(name="weights_11008x4096", op="weights", batch=0, n=11008, k=4096, codebook="e8p"),
    ]


def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + step)))
    return min(hi, max(lo, int(v) // step * step))


def draw(rng):
    """One more case of the ranges above: batch 1..2048 (64 for the stack and the integer operator), N in steps
    of 16 and K in steps of 32, stacks from a 1B to the 70B model's width."""
    op = rng.choices(["linear", "stack", "int8", "int8_inplace", "weights"], [6, 3, 2, 1, 1])[0]
    codebook = rng.choice(["synthetic", "e8p"])
    if op == "stack":
        hidden = _log(rng, 2048, 8192, 128)
        cfg = dict(hidden=hidden, kv_heads=rng.choice([8, hidden // 128]), head_dim=128,
                   ffn=_log(rng, 2 * hidden, 7 * hidden // 2, 32), layers=rng.randint(8, 80))
        return dict({"op": op, "batch": _log(rng, 1, 64), "codebook": codebook}, **cfg)
    while True:
        case = dict(op=op, batch=_log(rng, 1, 2048 if op == "linear" else 64), n=_log(rng, 512, 57344, 16),
                    k=_log(rng, 1024, 28672, 32), codebook=codebook)
        if op == "int8_inplace":
            case["n"] = case["n"] // 32 * 32  # its layout holds the rows in blocks of 32
        if op == "weights":
            case["batch"] = 0
        if max(case["batch"], 16) * case["n"] * case["k"] <= 2048 * 8192 * 28672:
            return case


def _codebook(case):
    if case["codebook"] == "e8p":
        return dmm.build_codebook_abs("cuda")
    return dmm.pack_codebook(dmm.synthetic_codebook(42)).to("cuda")


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op, batch = case["op"], case["batch"]
    cb64 = _codebook(case)
    if op == "stack":
        cfg = {key: case[key] for key in ("hidden", "kv_heads", "head_dim", "ffn", "layers")}
        stack = LinearStack(cfg, dmm.codebook_to_fp16(cb64), "cuda", seed=seed, scale=SCALE)
        return {"op": op, "stack": stack, "tokens": torch.randn(batch, case["hidden"], device="cuda", generator=gen)}
    n, k = case["n"], case["k"]
    codes = torch.randint(-32768, 32768, (n, k // 8), dtype=torch.int16, device="cuda", generator=gen)
    if op == "linear":
        x = torch.randn(batch, k, device="cuda", generator=gen).to(torch.float16)
        return {"op": op, "layer": DecodeLinear(codes, dmm.codebook_to_fp16(cb64), SCALE), "x": x}
    if op == "weights":
        return {"op": op, "codes": dmm.transpose_tile(codes), "codebook": dmm.codebook_to_fp16(cb64)}
    x = torch.randint(-128, 128, (batch, k), dtype=torch.int8, device="cuda", generator=gen)
    state = {"op": op, "x": x, "codebook": cb64}
    if op == "int8":
        return dict(state, codes=dmm.transpose_tile(codes))
    bias = torch.randint(-1000, 1000, (batch, n), dtype=torch.int32, device="cuda", generator=gen)
    return dict(state, codes=dmm.fast_pack(codes), bias=bias)


def run(state):
    op = state["op"]
    if op == "linear":
        return state["layer"](state["x"])
    if op == "stack":
        return state["stack"].step(state["tokens"].clone())  # the step works in place on the residual stream
    if op == "int8":
        return decode_matmul_int8(state["x"], state["codes"], state["codebook"])
    if op == "int8_inplace":
        return decode_matmul_int8_inplace(state["x"], state["codes"], state["codebook"], state["bias"].clone())
    return dmm.decode_weights(state["codes"], state["codebook"])


def work(case):
    op, batch = case["op"], case["batch"]
    if op == "stack":
        cfg = [case[key] for key in ("hidden", "kv_heads", "head_dim", "ffn")]
        weights = case["layers"] * sum(n * k for n, k in llama_shapes(*cfg).values())
        return {"bytes": weights // 4 + 4096 + 8 * batch * case["hidden"], "flops": 2 * batch * weights}
    n, k = case["n"], case["k"]
    if op == "weights":
        return {"bytes": n * k // 4 + 4096 + 2 * n * k, "flops": 0}
    x_bytes, out_bytes, table = {"linear": (2, 4, 4096), "int8": (1, 4, 2048), "int8_inplace": (1, 8, 2048)}[op]
    return {"bytes": n * k // 4 + table + x_bytes * batch * k + out_bytes * batch * n, "flops": 2 * batch * n * k}


def tolerance(case):
    # Against the same products in 64 bits a linear layer is off by 7.5e-7, or by up to 1.6e-6 with fp16 tensor-core
    # operands and other sums; a stack of blocks by up to 8.1e-6, because a sum that comes out one bit lower can
    # round to another half for the next product.  Four times that.
    if case["op"] == "linear":
        return {"rel": 6e-6}
    if case["op"] == "stack":
        return {"rel": 3.2e-5}
    return "exact"  # whole numbers, and halves that are copied out of a table
