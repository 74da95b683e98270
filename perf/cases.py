"""Workloads of the packed MoE layer as its users run them, for timing.

A case is a plain dict; ``prepare`` makes what a program holds before the call (packed layer or block, activations),
``run`` is one pass through the public entry points, ``work`` the traffic and arithmetic no implementation can avoid.

Four entry points are covered:

  block   a drop-in MoE block inside a decoder layer: ``block(hidden_states)`` with the router Linear (and the gated
          shared expert of Qwen3-Next) inside; what a patched Hugging Face model calls 48 times per step
  layer   ``PackedLayer.forward`` on router logits, with ``dense_mlp`` for the two shared experts of DeepSeek-V2-Lite
  op      ``moe_packed_forward``: the 26-argument op at the rank-space boundary, called with the block's buffer tuples
  pack    ``pack_single_weight``: the offline quantise-and-pack step of one expert matrix

The shapes are the three of ``bitsmoe_b200.synth`` with their mixed 2/3/4-bit allocations.  Decode batches go from one
sequence to a few hundred, prefill chunks to 16384 tokens; ``skew`` is the exponent of the Zipf law of the expert load.
"""
from types import SimpleNamespace
import math

import torch
import torch.nn as nn

from bitsmoe_b200 import synth
from bitsmoe_b200.algorithms import mlp_forward_cuda
from bitsmoe_b200.layer import PackedLayer, dense_mlp, route_build, route_topk
from bitsmoe_b200.models.qwen3moe.bitsmoe_block import BitsMoE_Qwen3MoeSparseMoeBlock
from bitsmoe_b200.models.qwen3moe.bitsmoe_mlp import BitsMoE_Qwen3MoeMLP
from bitsmoe_b200.models.qwen3next.bitsmoe_block import BitsMoE_Qwen3NextSparseMoeBlock
from bitsmoe_b200.models.qwen3next.bitsmoe_mlp import BitsMoE_Qwen3NextMLP
from bitsmoe_b200.quant.packer import pack_single_weight

DEVICE = "cuda"
QWEN, NEXT, DSV2 = synth.QWEN3_30B.name, synth.QWEN3_NEXT_80B.name, synth.DEEPSEEK_V2_LITE.name
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
MAX_TOKENS = {QWEN: 16384, NEXT: 16384, DSV2: 8192}


def listed():
    return [
        # one sequence being decoded: launches and host work are what counts
        {"name": "block_qwen3_1", "kind": "block", "shape": QWEN, "tokens": 1, "dtype": "bf16", "skew": 0.0},
        # the decode batch of the headline number
        {"name": "block_qwen3_64", "kind": "block", "shape": QWEN, "tokens": 64, "dtype": "bf16", "skew": 0.0},
        # a large decode batch of a busy server, not a multiple of anything
        {"name": "layer_qwen3_203", "kind": "layer", "shape": QWEN, "tokens": 203, "dtype": "fp16", "skew": 0.0},
        # one chunk of a chunked prefill with some decode tokens mixed in
        {"name": "block_qwen3_777", "kind": "block", "shape": QWEN, "tokens": 777, "dtype": "bf16", "skew": 0.8},
        # the prefill batch of the benchmark: Zipf(1.1) expert load
        {"name": "layer_qwen3_8192", "kind": "layer", "shape": QWEN, "tokens": 8192, "dtype": "bf16", "skew": 1.1},
        # decode on the layer with the most experts, gated shared expert included
        {"name": "block_next_24", "kind": "block", "shape": NEXT, "tokens": 24, "dtype": "bf16", "skew": 0.0},
        # long prefill on the same layer, the largest case
        {"name": "block_next_16384", "kind": "block", "shape": NEXT, "tokens": 16384, "dtype": "bf16", "skew": 0.5},
        # small decode batch of the uniform 2-bit layer with two shared experts
        {"name": "layer_deepseek_5", "kind": "layer", "shape": DSV2, "tokens": 5, "dtype": "fp16", "skew": 0.0},
        # one evaluation sequence of 2048 fp16 tokens, as the perplexity runs feed it
        {"name": "layer_deepseek_2048", "kind": "layer", "shape": DSV2, "tokens": 2048, "dtype": "fp16", "skew": 0.5},
        # the op on its own, where the caller keeps its own router and dense products
        {"name": "op_qwen3_48", "kind": "op", "shape": QWEN, "tokens": 48, "dtype": "fp16", "skew": 0.0},
        # one matrix of an expert on its way into a checkpoint
        {"name": "pack_qwen3", "kind": "pack", "shape": QWEN, "rank": 256, "dim": 768},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "layer", "layer", "layer", "op", "pack"])
    if kind == "pack":
        return {"kind": kind, "shape": QWEN, "rank": 8 * rng.randint(8, 64), "dim": 32 * rng.randint(8, 44)}
    shape = rng.choice([QWEN, QWEN, NEXT] if kind == "block" else [QWEN, DSV2, DSV2] if kind == "layer" else [QWEN, DSV2])
    tokens = _log_uniform(rng, 1, MAX_TOKENS[shape])
    return {"kind": kind, "shape": shape, "tokens": tokens, "dtype": "fp16" if kind == "op" else rng.choice(["bf16", "fp16"]),
            "skew": 0.0 if tokens <= 256 else round(rng.uniform(0.0, 1.1), 2)}


def _log_load(cfg, skew):
    p = 1.0 / torch.arange(1, cfg.num_experts + 1, device=DEVICE, dtype=torch.float32) ** skew
    return torch.log(p / p.sum())


class _DenseMLP(nn.Module):
    """The SwiGLU module a model carries as its shared expert."""

    def __init__(self, w, dtype):
        super().__init__()
        for name in ("gate", "up", "down"):
            lin = nn.Linear(w[name].shape[1], w[name].shape[0], bias=False, device="meta")
            lin.weight = nn.Parameter(w[name].to(dtype), requires_grad=False)
            setattr(self, name + "_proj", lin)

    def forward(self, x):
        return self.down_proj(nn.functional.silu(self.gate_proj(x)) * self.up_proj(x))


def _linear(weight):
    lin = nn.Linear(weight.shape[1], weight.shape[0], bias=False, device="meta")
    lin.weight = nn.Parameter(weight, requires_grad=False)
    return lin


def _activations(cfg, tokens, skew, seed, dtype):
    """N(0, 1) rows and a router weight that gives N(0, 1) logits; a skewed load comes, as it does in trained models,
    from a channel that has the same large value in every token."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed + 77)
    x = torch.randn(tokens, cfg.hidden, generator=gen, device=DEVICE)
    gate = torch.randn(cfg.num_experts, cfg.hidden, generator=gen, device=DEVICE) / math.sqrt(cfg.hidden)
    x[:, 0] = 8.0
    gate[:, 0] = _log_load(cfg, skew) / 8.0
    return x.to(dtype), gate.to(dtype)


def _build_block(cfg, layer, gate, dtype):
    block_cls, mlp_cls = ((BitsMoE_Qwen3NextSparseMoeBlock, BitsMoE_Qwen3NextMLP) if cfg.shared_intermediate else
                          (BitsMoE_Qwen3MoeSparseMoeBlock, BitsMoE_Qwen3MoeMLP))
    conf = SimpleNamespace(hidden_size=cfg.hidden, intermediate_size=cfg.intermediate, num_experts=cfg.num_experts,
                           num_experts_per_tok=cfg.top_k, norm_topk_prob=cfg.norm_topk_prob, hidden_act="silu")
    src = SimpleNamespace(gate=_linear(gate), experts=[None] * cfg.num_experts)
    if cfg.shared_intermediate:
        src.shared_expert = _DenseMLP(layer.shared, dtype)
        src.shared_expert_gate = _linear(layer.shared["gate_logit_w"].to(dtype))
    block = block_cls(conf, 0, src, copy_source_experts=False).eval()
    for e in range(cfg.num_experts):
        block.set_expert(e, mlp_cls(conf, cfg.intermediate, packed_state=layer.expert_state_dict(e, "e"), packed_prefix="e",
                                    packed_device=torch.device(DEVICE)), packed=True)
    block.set_shared_basis(layer.vh_gate, layer.vh_up, layer.u_down)
    block.prepare_runtime_fastpath(warmup=True)
    return block


def prepare(case, seed):
    if case["kind"] == "pack":
        gen = torch.Generator(device=DEVICE).manual_seed(seed)
        rank, dim = case["rank"], case["dim"]
        matrix = torch.randn(rank, dim, generator=gen, device=DEVICE) * 0.02
        s = torch.sort(torch.randn(rank, generator=gen, device=DEVICE).abs() + 0.05, descending=True).values
        # wide rows first: about 5 % of 4 bits, 15 % of 3 bits, the rest 2 bits, at boundaries that are not aligned
        a, b = max(1, rank // 20), max(2, rank // 5)
        segments = [(4, (0, a)), (3, (a, b)), (2, (b, rank))]
        return {"case": case, "moe": {0: {0: {"gate_proj": (matrix, s)}}}, "segments": segments}
    cfg = synth.PRESETS[case["shape"]]
    dtype, tokens, skew = DTYPES[case["dtype"]], case["tokens"], case["skew"]
    layer = synth.make_layer(cfg, seed=seed, device=DEVICE, keep_full=case["kind"] == "block")
    x, gate = _activations(cfg, tokens, skew, seed, dtype)
    state = {"case": case, "cfg": cfg, "x": x}
    if case["kind"] == "block":
        state["x"] = x.reshape(1, tokens, cfg.hidden) if tokens > 256 else x.reshape(tokens, 1, cfg.hidden)
        state["block"] = _build_block(cfg, layer, gate, dtype)
    elif case["kind"] == "layer":
        t = layer.tables
        state["layer"] = PackedLayer(t["gate"], t["up"], t["down"], cfg.intermediate, cfg.rank, layer.vh_gate, layer.vh_up, layer.u_down)
        state["shared"] = layer.shared
        # the logits a router hands over in fp32
        gen = torch.Generator(device=DEVICE).manual_seed(seed + 78)
        state["logits"] = torch.randn(tokens, cfg.num_experts, generator=gen, device=DEVICE) + _log_load(cfg, skew)
    else:
        gen = torch.Generator(device=DEVICE).manual_seed(seed + 78)
        logits = torch.randn(tokens, cfg.num_experts, generator=gen, device=DEVICE) + _log_load(cfg, skew)
        idx, w = route_topk(logits, cfg.top_k, cfg.norm_topk_prob, torch.float16)
        tok, off, rw, _, _ = route_build(idx, w, cfg.num_experts)
        h = torch.randn(2, tokens, cfg.rank, generator=gen, device=DEVICE).half()
        lists = [tuple(b.to(DEVICE) for b in layer.tables[tag][f]) for tag in ("gate", "up", "down")
                 for f in ("payload", "rank_idx", "tile_meta", "slab_meta", "scale", "s")]
        state["args"] = (h[0], h[1], tok, off, rw, *lists, cfg.rank, cfg.intermediate, 0)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pack":
        out = {}
        pack_single_weight(state["moe"], state["segments"], out, 0, 0, "gate_proj")
        return out
    if kind == "op":
        return mlp_forward_cuda.moe_packed_forward(*state["args"])
    with torch.inference_mode():
        if kind == "block":
            return state["block"](state["x"])
        cfg, sh = state["cfg"], state["shared"]
        x = state["x"]
        residual = dense_mlp(x, sh["gate"], sh["up"], sh["down"]) if sh else None
        return state["layer"].forward(x, state["logits"], cfg.top_k, cfg.norm_topk_prob,
                                      x.dtype if cfg.round_route_weights else None, residual=residual)


def _active_experts(cfg, tokens, skew):
    """Expected number of experts with at least one token when a token takes top_k of the skewed distribution."""
    p = [1.0 / (i + 1) ** skew for i in range(cfg.num_experts)]
    total = sum(p)
    return sum(1.0 - max(0.0, 1.0 - min(1.0, cfg.top_k * v / total)) ** tokens for v in p)


def work(case):
    if case["kind"] == "pack":
        n = case["rank"] * case["dim"]
        # factor read once; payload and scales written once; per weight and refinement round a divide, a rounding, two sums
        return {"bytes": 4 * n + n * 2.25 / 8 + n / 64, "flops": 50 * 6 * n}
    cfg = synth.PRESETS[case["shape"]]
    T, H, r, I, k = case["tokens"], cfg.hidden, cfg.rank, cfg.intermediate, cfg.top_k
    bits = sum(b * p for b, p in cfg.bit_probs)
    expert = 3 * (r * I * bits / 8 + r * (I / 128) * 2 + r * 6)
    nbytes = _active_experts(cfg, T, case["skew"]) * expert
    flops = T * k * 3 * 2 * r * I
    if case["kind"] == "op":
        return {"bytes": nbytes + T * r * 8 + T * k * 8, "flops": flops}
    nbytes += 3 * r * H * 2 + 2 * T * H * 2
    flops += T * 3 * 2 * H * r
    if case["kind"] == "block":
        nbytes += cfg.num_experts * H * 2 + T * cfg.num_experts * 2
        flops += T * 2 * H * cfg.num_experts
    else:
        nbytes += T * cfg.num_experts * 4
    if cfg.shared_intermediate:
        nbytes += 3 * H * cfg.shared_intermediate * 2
        flops += T * 3 * 2 * H * cfg.shared_intermediate
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "pack":
        return "exact"
    if case["kind"] == "block":
        # the router's logits are rounded to 16 bits: where two experts tie at the last place of a token's top-k another
        # summation order may take the other one, which moves single elements of that token but not the norm
        return {"rel": 1e-2, "max": 0.8}
    # operands are rounded to fp16 and summed in fp32
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 3e-3}
