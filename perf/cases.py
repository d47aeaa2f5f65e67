"""Performance cases of the framework on one GPU: what its users call, over the range they call it with.

Four entry points are covered:

* ``moe_forward``  ``models.moe_all2all.custom_kernel``: dispatch -> expert op of the task -> combine;
* ``moe_layer``    ``MoEAllToAll.dispatch`` and ``.combine`` around the caller's own experts;
* ``gemm_rs``      ``models.gemm_rs.custom_kernel``: row-parallel linear layer (one rank: GEMM + bias);
* ``fp8_gemm``     ``ops.fp8_gemm.fp8_gemm``: block-scaled fp8 GEMM.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes what a
program holds before the call, ``run`` is one call, ``work`` the bytes and operations the call cannot do
without and ``tolerance`` how far another correct implementation may be from the result.
"""
import math

import torch

from amd_distributed_2025_b200 import contract
from amd_distributed_2025_b200.models import gemm_rs, moe_all2all
from amd_distributed_2025_b200.ops.fp8_gemm import fp8_gemm

_DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32}
_SIZES = {"float16": 2, "bfloat16": 2, "float32": 4}

# The largest expert buffer (experts x tokens x hidden, in bytes) and the largest GEMM (2 M N K) of the
# listed cases: drawn ones stay below.
_MAX_EXPERT_BYTES = 64 * 4096 * 4096 * 2
_MAX_FLOPS = 2 * 8192 * 8192 * 28672
_MAX_FP8_FLOPS = 2 * 8192 * 8192 * 8192


def _moe(name, op, experts, topk, hidden, max_tokens, tokens, dtype, routing="uniform", weights="softmax"):
    return {"name": name, "op": op, "experts": experts, "topk": topk, "hidden": hidden, "max_tokens": max_tokens,
            "tokens": tokens, "dtype": dtype, "routing": routing, "weights": weights}


def _gemm(name, op, m, n, k, bias=False):
    return {"name": name, "op": op, "m": m, "n": n, "k": k, "bias": bias}


def listed():
    return [
        # The smallest decode step of the task's benchmark list (configs/all2all.yml): a dozen tokens, few wide
        # rows, fp16 with unnormalised weights.  Launches and host time are all there is.
        _moe("moe_forward_tiny_fp16", "moe_forward", 8, 2, 6144, 16, 11, "float16", weights="rand"),
        # Headline decode step (configs/headline.yml): many experts, a token or a few for each of them.
        _moe("moe_forward_decode_bf16", "moe_forward", 256, 8, 7168, 128, 128, "bfloat16"),
        # Headline prefill (configs/headline.yml): thousands of tokens with skewed routing.
        _moe("moe_forward_prefill_bf16", "moe_forward", 64, 6, 4096, 4096, 4096, "bfloat16", routing="zipf"),
        # The fp32 configuration of configs/headline.yml, as a layer around the caller's experts.
        _moe("moe_layer_tiny_fp32", "moe_layer", 16, 2, 256, 32, 32, "float32"),
        # A serving step of the task's benchmark list: odd token count below the layer's maximum.
        _moe("moe_layer_decode_fp16", "moe_layer", 128, 4, 2880, 128, 101, "float16", weights="rand"),
        # Prefill through the layer API: every token's rows out to the experts and back.
        _moe("moe_layer_prefill_bf16", "moe_layer", 128, 8, 4096, 2048, 2047, "bfloat16"),
        # The smallest linear layer of the task's test list, one rank's eighth of K: ragged in M, N and K.
        _gemm("gemm_rs_64x2880x360", "gemm_rs", 64, 2880, 360, True),
        # Decode-sized projection with a large weight (configs/gemm_rs.yml): the weight has to stream once.
        _gemm("gemm_rs_64x7168x18432", "gemm_rs", 64, 7168, 18432),
        # Headline sweep, small end (configs/headline.yml).
        _gemm("gemm_rs_256x5120x12800", "gemm_rs", 256, 5120, 12800, True),
        # Square, ragged against every tile width (configs/gemm_rs.yml).
        _gemm("gemm_rs_2048x2880x2880", "gemm_rs", 2048, 2880, 2880, True),
        # Headline training-sized layer (configs/headline.yml).
        _gemm("gemm_rs_8192x8192x28672", "gemm_rs", 8192, 8192, 28672, True),
        # Block-scaled fp8 GEMM at the size its tests end with.
        _gemm("fp8_gemm_4096x4096x2048", "fp8_gemm", 4096, 4096, 2048),
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread evenly over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(-(-lo // step) * step, int(v) // step * step)


def draw(rng):
    op = rng.choice(["moe_forward", "moe_forward", "moe_layer", "moe_layer", "gemm_rs", "gemm_rs", "gemm_rs", "fp8_gemm"])
    if op.startswith("moe"):
        dtype = rng.choice(["bfloat16", "bfloat16", "float16", "float16", "float32"])
        experts = _log_int(rng, 8, 256)
        topk = rng.randint(1, 8)
        hidden = _log_int(rng, 256, 7168, 8)  # rows are whole 16-byte vectors, not always whole tiles
        most = max(1, min(4096, _MAX_EXPERT_BYTES // (experts * hidden * _SIZES[dtype])))
        tokens = _log_int(rng, 1, most)
        # a layer is made for the largest batch it will see; this call brings that many tokens or fewer
        max_tokens = min(most, tokens + rng.randint(0, tokens))
        return {"op": op, "experts": experts, "topk": topk, "hidden": hidden, "max_tokens": max_tokens, "tokens": tokens,
                "dtype": dtype, "routing": rng.choice(["uniform", "zipf"]), "weights": rng.choice(["softmax", "rand"])}
    if op == "gemm_rs":
        m, n, k = _log_int(rng, 1, 8192), _log_int(rng, 512, 8192, 8), _log_int(rng, 256, 29568, 8)
        return {"op": op, "m": m, "n": n, "k": min(k, _MAX_FLOPS // (2 * m * n) // 8 * 8), "bias": rng.random() < 0.5}
    m, n, k = _log_int(rng, 16, 8192), _log_int(rng, 128, 8192, 8), _log_int(rng, 256, 8192, 16)
    return {"op": op, "m": m, "n": n, "k": min(k, _MAX_FP8_FLOPS // (2 * m * n) // 16 * 16), "bias": False}


def prepare(case, seed):
    op = case["op"]
    if op.startswith("moe"):
        cfg, data, rank, world = contract.make_moe_inputs(
            case["experts"], case["topk"], case["hidden"], case["max_tokens"], seed, 0, 1, device="cuda",
            dtype=_DTYPES[case["dtype"]], fixed_num_tokens=case["tokens"], routing=case["routing"], weights=case["weights"])
        layer = moe_all2all.get_layer(cfg, rank, world)
        if op == "moe_forward":
            return {"op": op, "input": (cfg, data, rank, world), "layer": layer}
        # Dispatch fills only the rows that tokens were sent to: the layer's buffers start out empty, as new ones do.
        layer.expert_x.zero_()
        layer.expert_meta.zero_()
        # The experts' own kernels are the caller's; their output is at hand in the dispatch layout.
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        expert_y = torch.empty_like(layer.expert_x).normal_(generator=gen)
        out = torch.empty((case["tokens"], case["hidden"]), dtype=cfg.out_dtype, device="cuda")
        return {"op": op, "layer": layer, "data": data, "expert_y": expert_y, "out": out}
    if op == "gemm_rs":
        a, w, bias = contract.make_gemm_rs_inputs(0, 1, case["m"], case["n"], case["k"], case["bias"], seed, device="cuda")
        gemm_rs.reserve([(case["m"], case["n"], case["k"])])  # the workspace, as a program makes it at start-up
        return {"op": op, "input": (a, w, bias)}
    m, n, k = case["m"], case["n"], case["k"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(m, k, device="cuda", generator=gen).to(torch.float8_e4m3fn)
    b = torch.randn(n, k, device="cuda", generator=gen).to(torch.float8_e4m3fn)
    a_scale = torch.rand(m, (k + 127) // 128, device="cuda", generator=gen) + 0.5
    b_scale = torch.rand((n + 127) // 128, (k + 127) // 128, device="cuda", generator=gen) + 0.5
    return {"op": op, "input": (a, b, a_scale, b_scale)}


def run(state):
    op = state["op"]
    if op == "moe_forward":
        return moe_all2all.custom_kernel(state["input"])
    if op == "moe_layer":
        layer, data = state["layer"], state["data"]
        counts, expert_x, meta = layer.dispatch(data.x, data.indices)
        layer.combine(state["out"], data.weights, meta, state["expert_y"], counts, data.num_tokens)
        return {"counts": counts, "expert_x": expert_x, "meta": meta, "out": state["out"]}
    if op == "gemm_rs":
        return gemm_rs.custom_kernel(state["input"])
    return fp8_gemm(*state["input"])


def work(case):
    if case["op"].startswith("moe"):
        tokens, entries = case["tokens"], case["tokens"] * case["topk"]
        row = case["hidden"] * _SIZES[case["dtype"]]
        total = 2 * tokens * row + entries * 8  # tokens in, result out, expert ids and weights
        if case["op"] == "moe_layer":
            # rows out to the experts and their results back in; 5 words of metadata a row, a count an expert
            total += 2 * entries * row + entries * 20 + case["experts"] * 4
        return {"bytes": total, "flops": 2 * entries * case["hidden"]}
    m, n, k = case["m"], case["n"], case["k"]
    if case["op"] == "gemm_rs":
        return {"bytes": 2 * (m * k + n * k + m * n) + (2 * n if case["bias"] else 0), "flops": 2 * m * n * k}
    kb = (k + 127) // 128
    return {"bytes": m * k + n * k + 2 * m * n + 4 * kb * (m + (n + 127) // 128), "flops": 2 * m * n * k}


def tolerance(case):
    # fp32 sums of a few terms; one or two roundings to the output type elsewhere.  Counts, metadata and
    # dispatched rows are copies and compare exactly within the same bound.
    if case["op"].startswith("moe"):
        return {"rel": {"float32": 1e-5, "float16": 2e-3, "bfloat16": 1e-2}[case["dtype"]]}
    return {"rel": 1e-2}
