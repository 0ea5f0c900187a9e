"""Performance cases of the MoE layer and of the operators around it.

Three kinds of work, each through the operators a serving engine calls:

``layer``   router logits and hidden states in; top-k routing, then ``fused_experts_impl``.
            One pass is one MoE layer of one forward step.
``align``   ``moe_align_block_size`` on its own, for engines that bring their own expert GEMM.
``router``  ``router_gemm``: the gate in front of the layer.

Shapes and value distributions are those of ``bench.py`` and ``flaggems_vllm_b200/testing.py``:
activations and logits ~N(0, 1), weights ~N(0, 0.02), routing bias ~N(0, 0.1)."""

from __future__ import annotations

import math

import torch

import flaggems_vllm_b200 as fg
from flaggems_vllm_b200 import testing

# experts, experts per token, hidden size, intermediate size
_SHAPES = {
    "dsv3": {"E": 256, "topk": 8, "H": 7168, "I": 2048},
    "mixtral": {"E": 8, "topk": 2, "H": 4096, "I": 14336},
    "qwen3": {"E": 128, "topk": 8, "H": 2048, "I": 768},
    "small": {"E": 8, "topk": 2, "H": 1024, "I": 2048},
}
# what the weights of each shape are stored as: e4m3 with 128x128 block scales, the activation type,
# weight-only int8, e4m3 or int8 with one scale per output channel and per token
_FORMATS = {
    "dsv3": ("fp8_block",),
    "mixtral": ("half",),
    "qwen3": ("int8_weight", "fp8_channel", "int8_channel"),
    "small": ("half",),
}
_MAX_TOKENS = {"fp8_block": 8192, "half": 16384, "int8_weight": 8192, "fp8_channel": 2048, "int8_channel": 2048}


def _layer(shape, fmt, tokens, dtype="bf16", ranks=1):
    return {"kind": "layer", "shape": shape, "format": fmt, "tokens": tokens, "dtype": dtype, "ranks": ranks}


def listed():
    return [
        # one sequence being decoded: latency and launches
        {"name": "dsv3_fp8_decode_1", **_layer("dsv3", "fp8_block", 1)},
        # a decode batch that fills no power of two: the weights of most experts are streamed
        {"name": "dsv3_fp8_decode_61", **_layer("dsv3", "fp8_block", 61)},
        # one rank of an 8-GPU expert-parallel deployment: 32 of 256 experts local, the tokens of all ranks
        {"name": "dsv3_fp8_rank_2000", **_layer("dsv3", "fp8_block", 2000, ranks=8)},
        # a full prefill chunk
        {"name": "dsv3_fp8_prefill_8192", **_layer("dsv3", "fp8_block", 8192)},
        {"name": "mixtral_bf16_decode_1", **_layer("mixtral", "half", 1)},
        # a large decode batch / a short prompt: between streaming weights and tensor-core bound
        {"name": "mixtral_bf16_mixed_300", **_layer("mixtral", "half", 300)},
        {"name": "mixtral_bf16_prefill_16384", **_layer("mixtral", "half", 16384)},
        # weight-only int8: a decode batch and a prefill chunk
        {"name": "qwen3_int8w_decode_33", **_layer("qwen3", "int8_weight", 33)},
        {"name": "qwen3_int8w_prefill_4096", **_layer("qwen3", "int8_weight", 4096)},
        # checkpoints quantised per channel, activations quantised per token at run time
        {"name": "qwen3_fp8ch_mixed_500", **_layer("qwen3", "fp8_channel", 500)},
        # half of the assignments on four experts, as real traffic is skewed
        {"name": "align_hot_8192", "kind": "align", "tokens": 8192, "E": 256, "topk": 8, "block": 128, "hot": True},
        # the gate of a mixed batch
        {"name": "router_dsv3_200", "kind": "router", "shape": "dsv3", "tokens": 200},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(("layer", "align", "router"), (10, 1, 1))[0]
    if kind == "align":
        return {"kind": "align", "tokens": _log_int(rng, 1, 8192), "E": 256, "topk": 8,
                "block": rng.choice((64, 128)), "hot": rng.random() < 0.5}
    if kind == "router":
        return {"kind": "router", "shape": rng.choice(("dsv3", "mixtral", "qwen3")), "tokens": _log_int(rng, 1, 8192)}
    shape = rng.choices(("dsv3", "mixtral", "qwen3", "small"), (4, 3, 4, 1))[0]
    fmt = rng.choice(_FORMATS[shape])
    ranks = rng.choice((1, 1, 2, 4, 8)) if shape == "dsv3" else 1
    return _layer(shape, fmt, _log_int(rng, 1, _MAX_TOKENS[fmt]), dtype=rng.choice(("bf16", "bf16", "bf16", "f16")),
                  ranks=ranks)


_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}


def _fp8_channel_weights(E, N, K, dev, seed):
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    q = torch.empty((E, N, K), dtype=torch.float8_e4m3fn, device=dev)
    s = torch.empty((E, N, 1), dtype=torch.float32, device=dev)
    for e0 in range(0, E, 16):
        w = torch.randn((min(16, E - e0), N, K), generator=g, device=dev) * 0.02
        sc = w.abs().amax(dim=-1, keepdim=True).clamp(min=1e-10) / 448.0
        q[e0:e0 + 16] = (w / sc).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
        s[e0:e0 + 16] = sc
    return q, s


def _weights(fmt, dtype, E, N, K, dev, seed):
    if fmt == "fp8_block":
        return testing.make_fp8_block_weights(E, N, K, dev, seed=seed)
    if fmt == "half":
        return testing.make_half_weights(E, N, K, dev, seed=seed, dtype=dtype, chunk=2), None
    if fmt == "fp8_channel":
        return _fp8_channel_weights(E, N, K, dev, seed)
    return testing.make_int8_channel_weights(E, N, K, dev, seed=seed)


def prepare(case, seed):
    dev = torch.device("cuda")
    base = seed * 16
    if case["kind"] == "align":
        return {"case": case, "ids": testing.make_align_ids(case["tokens"], case["topk"], case["E"], dev,
                                                            skewed=case["hot"], seed=base)}
    c = _SHAPES[case["shape"]]
    M, E, H, I = case["tokens"], c["E"], c["H"], c["I"]
    if case["kind"] == "router":
        return {"case": case, "x": testing.make_activations(M, H, dev, seed=base + 1),
                "gate": testing.make_half_weights(1, E, H, dev, seed=base + 2)[0]}
    dtype = _DTYPES[case["dtype"]]
    local = E // case["ranks"]
    w1, s1 = _weights(case["format"], dtype, local, 2 * I, H, dev, base + 3)
    w2, s2 = _weights(case["format"], dtype, local, H, I, dev, base + 4)
    logits, bias = testing.make_router_inputs(M, E, dev, seed=base + 5)
    options = {"global_num_experts": E}
    if case["ranks"] > 1:
        first = local * (seed % case["ranks"])
        emap = torch.full((E,), -1, dtype=torch.int32, device=dev)
        emap[first:first + local] = torch.arange(local, dtype=torch.int32, device=dev)
        options["expert_map"] = emap
    if s1 is not None:
        options.update(w1_scale=s1, w2_scale=s2)
    options.update({"fp8_block": {"use_fp8_w8a8": True, "block_shape": [128, 128]}, "half": {},
                    "int8_weight": {"use_int8_w8a16": True, "per_channel_quant": True},
                    "fp8_channel": {"use_fp8_w8a8": True, "per_channel_quant": True},
                    "int8_channel": {"use_int8_w8a8": True, "per_channel_quant": True}}[case["format"]])
    return {"case": case, "x": testing.make_activations(M, H, dev, seed=base + 1, dtype=dtype), "w1": w1, "w2": w2,
            "logits": logits, "bias": bias, "options": options}


def run(state):
    case = state["case"]
    if case["kind"] == "align":
        return fg.moe_align_block_size(state["ids"], case["block"], case["E"])
    if case["kind"] == "router":
        return fg.router_gemm(state["x"], state["gate"])
    logits, topk = state["logits"], _SHAPES[case["shape"]]["topk"]
    if case["shape"] == "dsv3":
        weights, ids = fg.grouped_topk(logits, 8, 4, topk, True, 2.5, state["bias"], 1)
    else:
        # the caller of this operator owns the outputs
        M = logits.shape[0]
        weights = torch.empty((M, topk), dtype=torch.float32, device=logits.device)
        ids = torch.empty((M, topk), dtype=torch.int32, device=logits.device)
        rows = torch.empty((M, topk), dtype=torch.int32, device=logits.device)
        fg.topk_softmax(weights, ids, rows, logits, True)
    out = fg.fused_experts_impl(state["x"], state["w1"], state["w2"], weights, ids, **state["options"])
    return {"out": out, "weights": weights, "ids": ids}


def _experts_used(case, E, k):
    """Experts that get at least one token, from the distributions that ``prepare`` draws from."""
    M = case["tokens"]
    if case["shape"] != "dsv3":
        return E * (1.0 - (1.0 - k / E) ** M)  # even routing
    # the routing bias favours some experts of some groups: counted on two samples
    used = 0
    for sample in range(2):
        g = torch.Generator().manual_seed(sample)
        scores = torch.sigmoid(torch.randn((M, E), generator=g)) + 0.1 * torch.randn((E,), generator=g)
        groups = scores.view(M, 8, E // 8)
        best = groups.topk(2, dim=-1).values.sum(-1).topk(4, dim=-1).indices
        open_ = torch.zeros((M, 8)).scatter_(1, best, 1.0).bool().repeat_interleave(E // 8, dim=1)
        used += scores.masked_fill(~open_, -1.0).topk(k, dim=-1).indices.unique().numel()
    return used / 2


def work(case):
    M = case["tokens"]
    if case["kind"] == "align":
        numel, E, bs = M * case["topk"], case["E"], case["block"]
        padded = numel + E * (bs - 1)
        return {"bytes": 4 * (numel + padded + -(-padded // bs) + 1), "flops": 0}
    c = _SHAPES[case["shape"]]
    E, k, H, I = c["E"], c["topk"], c["H"], c["I"]
    if case["kind"] == "router":
        return {"bytes": 2 * (M * H + E * H) + 4 * M * E, "flops": 2 * M * E * H}
    used = _experts_used(case, E, k) / case["ranks"]
    width = 2 if case["format"] == "half" else 1
    weights = used * 3 * H * I * width
    if case["format"] == "fp8_block":
        weights += used * 3 * (H // 128) * (I // 128) * 4
    elif case["format"] != "half":
        weights += used * (2 * I + H) * 4
    return {"bytes": weights + 2 * M * H * 2 + M * E * 4 + M * k * 8,
            "flops": 6 * H * I * M * k / case["ranks"]}


def tolerance(case):
    if case["kind"] == "align":
        return "exact"
    if case["kind"] == "router":
        return {"rel": 1e-5}  # fp32 sums of exact bf16 products
    return {"rel": 1e-2}      # the intermediate is rounded to bf16 or 8 bits between the two GEMMs; ids are exact
