"""The measured workloads of the MoE-layer path, as a serving program runs them.

Five kinds of work, told apart by a case's ``kind``:

* ``layer``    one MoE block on activations that already sit in HBM, through
               `B200MoeBlock.forward_device`, replayed from a CUDA graph (``graph``:
               a serving loop with fixed buffers) or launched kernel by kernel
               (eager: a loop whose batch changes every step);
* ``block``    the same block through `B200MoeBlock.forward` on ``[batch, seq,
               hidden]``, the contract of the block it is plugged in for: returns
               the rows and the router logits;
* ``host``     one batch from pinned host memory and back, `forward_host`;
* ``decode``   one step of the whole shaped model (`ShapedMoeModel.decode_step`:
               attention over the cache, norms, MoE block of every layer, lm_head);
* ``prefill``  the prompt pass of the whole shaped model (`ShapedMoeModel.prefill`).

Token counts run from one sequence's decode step to a 16384-token prefill batch,
over the two block shapes of `synth`, with the uniform routing of a plain router
and with the skewed routing of a Zipf(1.2) router bias.  Weights are N(0, 0.02),
activations N(0, 1), token ids uniform, all drawn on the GPU from the seed.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from sparse_b200 import synth
from sparse_b200.block import B200MoeBlock
from sparse_b200.model import DEEPSEEK_MODEL, QWEN_MODEL, ShapedMoeModel, random_layer_weights

SHAPES = {"qwen": synth.QWEN_MOE, "deepseek": synth.DEEPSEEK_V2_LITE}
# The deepseek shape runs with the first third of its layers, the share of one of
# three pipeline stages: over all 27 the rounding of bf16 sums in another order
# grows past what a comparison can tell from a mistake (3.6 % in the last cache).
MODELS = {"qwen": QWEN_MODEL, "deepseek": dataclasses.replace(DEEPSEEK_MODEL, layers=9)}
ZIPF_SEED = 7


def listed():
    return [
        # one sequence decoding: the weights of four experts and the shared one per token
        {"name": "layer_qwen_1", "kind": "layer", "shape": "qwen", "tokens": 1, "zipf": 1.2, "graph": True},
        # a small decode batch through the plug-in contract, launched eagerly
        {"name": "block_deepseek_8", "kind": "block", "shape": "deepseek", "batch": 8, "seq": 1, "zipf": 0.0},
        # a serving-sized decode batch: few rows for each of many experts
        {"name": "layer_qwen_64", "kind": "layer", "shape": "qwen", "tokens": 64, "zipf": 1.2, "graph": True},
        # a prefill chunk mixed with decodes: ragged, every expert hit
        {"name": "layer_deepseek_300", "kind": "layer", "shape": "deepseek", "tokens": 300, "zipf": 0.0,
         "graph": True},
        # one prompt of odd length through the plug-in contract
        {"name": "block_qwen_1x1003", "kind": "block", "shape": "qwen", "batch": 1, "seq": 1003, "zipf": 1.2},
        # the benchmark's batch: 4096 tokens, skewed routing
        {"name": "layer_qwen_4096", "kind": "layer", "shape": "qwen", "tokens": 4096, "zipf": 1.2, "graph": True},
        # a prefill batch that fills no tile evenly
        {"name": "block_deepseek_3x1667", "kind": "block", "shape": "deepseek", "batch": 3, "seq": 1667, "zipf": 0.0},
        # the largest prefill batch
        {"name": "layer_qwen_16384", "kind": "layer", "shape": "qwen", "tokens": 16384, "zipf": 0.0, "graph": False},
        # the benchmark's batch when it lives in host memory
        {"name": "host_qwen_4096", "kind": "host", "shape": "qwen", "tokens": 4096, "zipf": 1.2, "graph": True},
        # one generated token for each of eight sequences with 2048 cached positions
        {"name": "decode_qwen_8x2048", "kind": "decode", "shape": "qwen", "batch": 8, "context": 2048},
        # one sequence generating: latency of the whole model
        {"name": "decode_deepseek_1x1024", "kind": "decode", "shape": "deepseek", "batch": 1, "context": 1024},
        # the prompts of eight sequences
        {"name": "prefill_qwen_8x2048", "kind": "prefill", "shape": "qwen", "batch": 8, "context": 2048},
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["layer", "block", "host", "decode", "prefill"], [6, 5, 2, 2, 1])[0]
    shape = rng.choice(["qwen", "deepseek"])
    if kind in ("decode", "prefill"):
        context = _log_uniform(rng, 32, 2048)
        batch = _log_uniform(rng, 1, 16 if kind == "decode" else 8)
        return {"kind": kind, "shape": shape, "batch": batch, "context": context}
    zipf = rng.choice([0.0, 1.2])
    tokens = _log_uniform(rng, 1, 16384)
    if kind == "block":
        batch = min(tokens, rng.choice([1, 2, 3, 5, 8]))
        return {"kind": kind, "shape": shape, "batch": batch, "seq": tokens // batch, "zipf": zipf}
    return {"kind": kind, "shape": shape, "tokens": tokens, "zipf": zipf, "graph": rng.random() < 0.5}


def _tokens(case) -> int:
    return case["batch"] * case["seq"] if case["kind"] == "block" else case["tokens"]


def _block(case, seed: int, device) -> B200MoeBlock:
    shape = SHAPES[case["shape"]]
    weights = random_layer_weights(shape, device, seed, range(shape.num_experts))
    if case["zipf"] > 0:
        weights.set_router(weights.router_w, synth.zipf_router_bias(shape.num_experts, case["zipf"], ZIPF_SEED + seed))
    return B200MoeBlock(weights, shape.top_k, _tokens(case), norm_topk_prob=shape.norm_topk_prob,
                        fp32_router_logits=case["shape"] == "deepseek", use_graphs=case.get("graph", False))


def prepare(case, seed: int):
    device = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=device).manual_seed(seed + 17)
    if case["kind"] in ("decode", "prefill"):
        cfg, batch, context = MODELS[case["shape"]], case["batch"], case["context"]
        model = ShapedMoeModel(cfg, device, batch, context + 64, seed=seed)
        ids = torch.randint(0, cfg.vocab, (batch, context), generator=gen, device=device)
        state = {"case": case, "model": model, "ids": ids}
        if case["kind"] == "decode":
            # the prompt is in the cache and every sequence has its next token
            model.prefill(ids)
            state["next"] = torch.randint(0, cfg.vocab, (batch,), generator=gen, device=device)
        return state
    shape, tokens = SHAPES[case["shape"]], _tokens(case)
    x = torch.randn((tokens, shape.hidden), generator=gen, device=device).to(torch.bfloat16)
    state = {"case": case, "block": _block(case, seed, device)}
    if case["kind"] == "host":
        state["x"] = x.cpu().pin_memory()
        state["out"] = torch.empty_like(state["x"]).pin_memory()
    elif case["kind"] == "block":
        state["x"] = x.view(case["batch"], case["seq"], shape.hidden)
    else:
        state["x"], state["out"] = x, torch.empty_like(x)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "layer":
        out = state["block"].forward_device(state["x"], state["out"])
        return out, state["block"].topk(case["tokens"])
    if kind == "block":
        return state["block"].forward(state["x"])
    if kind == "host":
        state["block"].forward_host(state["x"], state["out"])
        return state["out"]
    model = state["model"]
    if kind == "prefill":
        logits = model.prefill(state["ids"])
        return logits, _cache(model, 0, case["context"])
    # as `greedy_decode_profiled` begins its loop after the prompt pass
    model.cur_ids.copy_(state["next"])
    model.cur_pos.fill_(case["context"])
    model.decode_step()
    # The keys and values that the step added to the cache of every layer.  (The
    # argmax of a random-init model has no margin: it is not compared.)
    return _cache(model, case["context"], 1)


def _cache(model, begin: int, length: int):
    return [(ly.cache_k.narrow(1, begin, length), ly.cache_v.narrow(1, begin, length)) for ly in model.layers]


@functools.lru_cache(maxsize=None)
def _hit_rate(shape_name: str, zipf: float):
    """Chance of each expert to be among a token's top-k (sampled once, fixed seed)."""
    shape = SHAPES[shape_name]
    logits = np.random.RandomState(0).standard_normal((4096, shape.num_experts)) * 0.02 * math.sqrt(shape.hidden)
    if zipf > 0:
        logits = logits + synth.zipf_router_bias(shape.num_experts, zipf, ZIPF_SEED).numpy()
    top = np.argpartition(-logits, shape.top_k, axis=1)[:, :shape.top_k]
    return np.bincount(top.reshape(-1), minlength=shape.num_experts) / 4096.0


def _moe_work(shape_name: str, tokens: int, zipf: float):
    """(weight bytes, flops) of one MoE block: the experts that `tokens` tokens hit, each read once."""
    shape = SHAPES[shape_name]
    hit = float((1.0 - (1.0 - _hit_rate(shape_name, zipf)) ** tokens).sum())
    weights = hit * shape.routed_expert_bytes_bf16 + 3 * shape.hidden * shape.shared_inter * 2
    return weights + (shape.num_experts + int(shape.shared_gate)) * shape.hidden * 2, shape.flops_per_token() * tokens


def work(case):
    if case["kind"] not in ("decode", "prefill"):
        shape, tokens = SHAPES[case["shape"]], _tokens(case)
        nbytes, flops = _moe_work(case["shape"], tokens, case["zipf"])
        rows = 2 * tokens * shape.hidden * 2                    # activations in and out
        small = tokens * (shape.top_k * 6 + shape.num_experts * (4 if case["shape"] == "deepseek" else 2))
        return {"bytes": nbytes + rows + small, "flops": flops}
    cfg, batch, context = MODELS[case["shape"]], case["batch"], case["context"]
    tokens = batch if case["kind"] == "decode" else batch * context
    nbytes = flops = 0.0
    for layer in range(cfg.layers):
        if layer in cfg.dense_layers:
            params = 3 * cfg.hidden * cfg.dense_layers[layer]
            nbytes, flops = nbytes + 2 * params, flops + 2 * params * tokens
        else:
            b, f = _moe_work(case["shape"], tokens, 0.0)
            nbytes, flops = nbytes + b, flops + f
    if cfg.attention == "mla":
        nope = cfg.qk_dim - cfg.rope_dim
        proj = (cfg.n_heads * cfg.qk_dim + cfg.kv_lora_rank + cfg.rope_dim) * cfg.hidden
        proj += cfg.n_heads * (nope + cfg.v_dim) * cfg.kv_lora_rank
    else:
        proj = (cfg.n_heads * cfg.qk_dim + cfg.n_kv_heads * (cfg.qk_dim + cfg.v_dim)) * cfg.hidden
    proj += cfg.hidden * cfg.n_heads * cfg.v_dim
    per_position = cfg.n_kv_heads * (cfg.qk_dim + cfg.v_dim) * 2                  # cache bytes of one position
    if case["kind"] == "decode":
        pairs, cached = batch * (context + 1), batch * (context + 1)
    else:
        pairs, cached = batch * context * (context + 1) / 2, batch * context
    nbytes += cfg.layers * (2 * proj + cached * per_position) + 2 * cfg.vocab * cfg.hidden
    flops += cfg.layers * (2 * proj * tokens + 2 * pairs * cfg.n_heads * (cfg.qk_dim + cfg.v_dim))
    flops += 2 * batch * cfg.vocab * cfg.hidden
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # Measured on a B200: the same rows through the weight-streaming and through the
    # tensor-core kernels (fp32 sums in another order) differ by 8.4e-4 (2-norm) and
    # 0.019 (largest, over the larger of the value and the root mean square); the
    # models, prompts cut into chunks of 16 tokens instead of 1024 to 2048, by 1.9e-2
    # (qwen, 24 layers; largest 0.4), since a changed rounding now and then changes
    # a token's set of experts.
    if case["kind"] in ("decode", "prefill"):
        return {"rel": 0.03, "max": 0.95}
    return {"rel": 0.0035, "max": 0.08}
