"""The work that a user of this library has it do, as cases that can be timed one by one.

Sizes: one layer is the fixed model shape (hidden 2048, 256 experts of intermediate 512, top-8, one shared
expert).  Prefill takes 1 .. 8192 rows per call (the handle's capacity in production), decode takes one row through
1 .. 40 layers, the LM head scans up to 248 320 rows, and the dense product is called with the projection shapes of the
same model.  Weights are BF16 N(0, 0.02) and activations BF16 N(0, 1); routing is that of random rows (uniform over
the experts), skewed along a Zipf ranking, sent to eight hot experts, or full of ties (logits in steps of 1/8).
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

aima = importlib.import_module("aima-amd395-qwen36-35b-linux-engine_b200")

HIDDEN, EXPERTS, TOP_K, INTER, SHARED = 2048, 256, 8, 512, 512
VOCAB = 248320
EXPERT_BYTES = 3 * INTER * HIDDEN * 2                    # gate, up and down of one expert
FIXED_BYTES = EXPERTS * HIDDEN * 2 + 3 * SHARED * HIDDEN * 2 + 2 * HIDDEN * 2   # router, shared expert, its gate, the norm
ROW_FLOPS = 2 * (EXPERTS * HIDDEN + HIDDEN + (TOP_K + 1) * 3 * INTER * HIDDEN)  # one row through one layer
MAX_DISTINCT = 20    # a stack of more layers binds the same 20 sets of weights again (1.6 GB each, all larger than L2)


def listed() -> list[dict]:
    return [
        # the smallest call: the MoE half of one layer for one token, between a host's own attention kernels
        {"name": "decode_layer", "kind": "decode_calls", "layers": 1},
        # the same as a host runs it for a token: one call per layer, each on the output of the one before
        {"name": "decode_calls_20", "kind": "decode_calls", "layers": 20},
        # one token through all 40 layers in one launch: the repository's own headline workload
        {"name": "decode_stack_40", "kind": "decode_stack", "layers": 40},
        # a short prompt, or the few rows left over at the end of a chunked one
        {"name": "prefill_16", "kind": "prefill", "tokens": 16, "routing": "uniform"},
        # an ordinary chat prompt of odd length
        {"name": "prefill_333", "kind": "prefill", "tokens": 333, "routing": "uniform"},
        # the smallest of the prefill buckets
        {"name": "prefill_1024", "kind": "prefill", "tokens": 1024, "routing": "uniform"},
        # one layer with the norms on either side of it, ragged row count: what a host calls between two attention halves
        {"name": "prefill_fused_2047", "kind": "prefill_fused", "tokens": 2047, "routing": "uniform"},
        # the stack entry on a middle bucket: four layers, norms between them
        {"name": "prefill_stack_4096x4", "kind": "prefill_stack", "tokens": 4096, "layers": 4, "routing": "uniform"},
        # the largest bucket: one chunk of a long prompt, balanced routing ...
        {"name": "prefill_8192", "kind": "prefill", "tokens": 8192, "routing": "uniform"},
        # ... and skewed routing (some experts with more than 1000 rows, many with fewer than 10)
        {"name": "prefill_8192_zipf", "kind": "prefill", "tokens": 8192, "routing": "zipf"},
        # the next token's id from the final hidden row, full vocabulary
        {"name": "lm_head_248320", "kind": "lm_head", "rows": VOCAB},
        # the dense product at the shape of the fused attention input projection of a full chunk
        {"name": "gemm_8192x12352x2048", "kind": "gemm", "m": 8192, "n": 12352, "k": 2048},
    ]


def _log_int(rng, low: int, high: int) -> int:
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng) -> dict:
    kind = rng.choice(["prefill"] * 5 + ["prefill_fused", "prefill_stack", "decode_calls", "decode_stack", "decode_stack", "lm_head", "gemm", "gemm"])
    if kind in ("prefill", "prefill_fused"):
        return {"kind": kind, "tokens": _log_int(rng, 1, 8192), "routing": rng.choice(["uniform", "uniform", "zipf", "zipf", "hot", "ties"])}
    if kind == "prefill_stack":
        tokens = _log_int(rng, 2, 4096)
        return {"kind": kind, "tokens": tokens, "layers": rng.randint(2, 4), "routing": rng.choice(["uniform", "zipf"])}
    if kind == "decode_calls":
        return {"kind": kind, "layers": rng.randint(2, 19)}
    if kind == "decode_stack":
        return {"kind": kind, "layers": rng.randint(2, 39)}
    if kind == "lm_head":
        return {"kind": kind, "rows": _log_int(rng, 8192, VOCAB)}
    # projections of the model: in and out of the attention half, shared expert, vocabulary slices; k as the GEMV entry's
    return {"kind": "gemm", "m": _log_int(rng, 1, 8192), "n": 8 * _log_int(rng, 32, 1544), "k": rng.choice([512, 2048, 4096])}


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(1_000_003 * seed + 17)


def _normal(generator: torch.Generator, *shape: int, std: float = 1.0) -> torch.Tensor:
    return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=generator)


def _provider(case: dict, seed: int, layers: int, capacity: int):
    """A handle with its layers bound: what a serving process builds once."""
    device = torch.device("cuda", torch.cuda.current_device())
    provider = aima.MoeProvider(layers=layers, max_prefill_tokens=capacity)
    distinct = _layer_weights(layers, seed)
    for layer in range(layers):
        provider.bind_layer(layer, distinct[layer % len(distinct)])
    routing = case.get("routing", "uniform")
    if routing == "zipf":
        provider.set_router_hooks(aima.synth.zipf_router_bias(seed).to(device))
    elif routing == "hot":
        provider.set_router_hooks(aima.synth.hot_expert_bias(range(3, EXPERTS, 32)).to(device))
    elif routing == "ties":
        provider.set_router_hooks(None, quantize_eighths=True)
    return provider


def _layer_weights(layers: int, seed: int) -> list:
    device = torch.device("cuda", torch.cuda.current_device())
    return [aima.synth.layer_weights_cuda_fast(seed, layer, device) for layer in range(min(layers, MAX_DISTINCT))]


def prepare(case: dict, seed: int) -> dict:
    kind, generator = case["kind"], _generator(seed)
    state = {"kind": kind}
    if kind in ("decode_calls", "decode_stack"):
        state["provider"] = _provider(case, seed, case["layers"], 0)
        state["layers"] = case["layers"]
        state["x"] = _normal(generator, HIDDEN)
        state["out"] = torch.empty_like(state["x"])
    elif kind in ("prefill", "prefill_fused", "prefill_stack"):
        tokens = case["tokens"]
        state["provider"] = _provider(case, seed, case.get("layers", 1), tokens)
        state["a"] = _normal(generator, tokens, HIDDEN)
        if kind == "prefill_stack":
            state["out"] = torch.empty_like(state["a"])
        else:
            state["b"] = _normal(generator, tokens, HIDDEN)
        if kind == "prefill_fused":
            state["next_norm"] = _normal(generator, HIDDEN, std=0.02)
    elif kind == "lm_head":
        state["head"] = aima.LmHead(_normal(generator, case["rows"], HIDDEN, std=0.02))
        state["hidden"] = _normal(generator, HIDDEN)
    else:
        state["provider"] = aima.MoeProvider(layers=1)
        state["a"] = _normal(generator, case["m"], case["k"])
        state["b"] = _normal(generator, case["n"], case["k"], std=0.02)
    return state


def run(state: dict):
    kind = state["kind"]
    if kind == "decode_calls":
        x = state["x"]
        for layer in range(state["layers"]):
            x = state["provider"].decode_layer(x, layer)
        return x
    if kind == "decode_stack":
        return state["provider"].decode_stack(state["x"], state["out"])
    if kind == "prefill":
        return state["provider"].launch_selected_moe(post_attention=state["a"], residual_hidden=state["b"], model_layer=0)
    if kind == "prefill_fused":
        return state["provider"].prefill_fused(state["a"], state["b"], 0, next_norm_weight=state["next_norm"])
    if kind == "prefill_stack":
        return state["provider"].prefill_stack(state["a"], state["out"])
    if kind == "lm_head":
        # the token id is needed on the host before the next step can start
        logits = state["head"].launch(state["hidden"])
        result = state["head"].result()
        return logits, result.exact_top1_token_id, result.exact_top1_logit
    return state["provider"].gemm(state["a"], state["b"])


def _experts_touched(case: dict) -> int:
    """Experts that at least one of the rows is routed to, from a simulated routing of the same distribution."""
    if case["routing"] == "hot":
        return TOP_K
    logits = np.random.RandomState(7).standard_normal((case["tokens"], EXPERTS)).astype(np.float32) * (0.02 * math.sqrt(HIDDEN))
    if case["routing"] == "zipf":
        logits += aima.synth.zipf_router_bias(7).numpy()
    return len(np.unique(np.argpartition(logits, EXPERTS - TOP_K, axis=1)[:, EXPERTS - TOP_K:]))


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("decode_calls", "decode_stack"):
        layers = case["layers"]
        return {"bytes": layers * (TOP_K * EXPERT_BYTES + FIXED_BYTES) + 2 * HIDDEN * 2, "flops": layers * ROW_FLOPS}
    if kind in ("prefill", "prefill_fused", "prefill_stack"):
        layers, tokens = case.get("layers", 1), case["tokens"]
        tensors = {"prefill": 3, "prefill_fused": 4, "prefill_stack": 2}[kind]
        return {"bytes": layers * (_experts_touched(case) * EXPERT_BYTES + FIXED_BYTES) + tensors * tokens * HIDDEN * 2,
                "flops": layers * tokens * ROW_FLOPS}
    if kind == "lm_head":
        # the int8 copy, a scale and a residual norm per row; the logits out
        return {"bytes": case["rows"] * (HIDDEN + 12) + HIDDEN * 2, "flops": 2 * case["rows"] * HIDDEN}
    m, n, k = case["m"], case["n"], case["k"]
    return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * n * k}


def tolerance(case: dict):
    kind = case["kind"]
    if kind in ("decode_calls", "decode_stack", "lm_head"):
        return "exact"       # one documented order of summation, checked bit for bit against the oracle
    # four times what the tensor-core products differ from CUDA-core ones that sum in another order: one layer
    # rel 2.6e-4 / max 1.3e-2 on every size and routing; a stack of four, where such a difference now and then moves a
    # row to another expert, rel 6e-3 / max 0.18
    if kind == "prefill_stack":
        return {"rel": 6.0e-3 * case["layers"], "max": 0.72}
    if kind == "gemm":
        return {"rel": 4.0e-3, "max": 0.016}      # one BF16 rounding: rel 1.7e-3 / max 3.9e-3 against FP64
    return {"rel": 1.1e-3, "max": 0.05}


# ---- the same values in 64 bits ----------------------------------------------------------------------------------

def _norm64(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    return x * torch.rsqrt((x * x).mean(dim=-1, keepdim=True) + 1.0e-6) * (1.0 + weight.double())


def _moe64(h: torch.Tensor, weights: dict, logit_hook) -> torch.Tensor:
    """routed + shared experts of one layer for the rows of h, everything but the routing decision unrounded."""
    logits = logit_hook(h @ weights["router"].double().T)
    order = torch.sort(logits, dim=1, descending=True, stable=True)           # ties: lowest expert first
    ids, share = order.indices[:, :TOP_K], torch.softmax(order.values[:, :TOP_K], dim=1)
    out = torch.zeros_like(h)
    for expert in torch.unique(ids).tolist():
        row, slot = torch.nonzero(ids == expert, as_tuple=True)
        gate, up = (h[row] @ weights["expert_gate_up"][expert].double().T).split(INTER, dim=1)
        down = (torch.nn.functional.silu(gate) * up) @ weights["expert_down"][expert].double().T
        out.index_add_(0, row, down * share[row, slot].unsqueeze(1))
    act = torch.nn.functional.silu(h @ weights["shared_gate_proj"].double().T) * (h @ weights["shared_up_proj"].double().T)
    return out + torch.sigmoid(h @ weights["shared_gate"].double().T) * (act @ weights["shared_down_proj"].double().T)


def exact(case: dict, seed: int):
    kind, generator = case["kind"], _generator(seed)
    if kind == "gemm":
        a = _normal(generator, case["m"], case["k"])
        return a.double() @ _normal(generator, case["n"], case["k"], std=0.02).double().T
    if kind == "lm_head":
        # the logits of the int8 copy; the few rows that are evaluated exactly move the norm by less than it is off
        weight, hidden = _normal(generator, case["rows"], HIDDEN, std=0.02), _normal(generator, HIDDEN).double()
        parts = []
        for rows in weight.split(16384):
            scale = rows.float().abs().amax(dim=1).clamp_min(1.0e-12) * np.float32(1.0 / 127.0)
            q = (rows.float() / scale.unsqueeze(1)).round().clamp(-127, 127)
            parts.append((q.double() @ hidden) * scale.double())
        return torch.cat(parts), None, None
    layers = case.get("layers", 1)
    if layers > 20:
        return None          # a token through that many layers of random weights: roundings decide its later experts
    weights = _layer_weights(layers, seed)
    if kind in ("decode_calls", "decode_stack"):
        x = _normal(generator, HIDDEN).double().unsqueeze(0)
        for layer in range(layers):
            w = weights[layer % len(weights)]
            x = x + _moe64(_norm64(x, w["post_attention_layernorm"]), w, lambda logits: logits)
        return x[0]
    routing, device = case.get("routing", "uniform"), weights[0]["router"].device
    bias = {"zipf": lambda: aima.synth.zipf_router_bias(seed).to(device),
            "hot": lambda: aima.synth.hot_expert_bias(range(3, EXPERTS, 32)).to(device)}.get(routing, lambda: 0.0)()

    def hook(logits: torch.Tensor) -> torch.Tensor:      # the path routes by BF16 logits
        logits = logits + bias
        if routing == "ties":
            logits = (logits * 8.0).round() * 0.125
        return logits.bfloat16().double()

    a = _normal(generator, case["tokens"], HIDDEN).double()
    if kind == "prefill_stack":
        for layer in range(layers):
            a = a + _moe64(_norm64(a, weights[layer]["post_attention_layernorm"]), weights[layer], hook)
        return a
    b = _normal(generator, case["tokens"], HIDDEN).double()
    if kind == "prefill":
        return b + _moe64(a, weights[0], hook)
    residual = a + b
    out = residual + _moe64(_norm64(residual, weights[0]["post_attention_layernorm"]), weights[0], hook)
    return out, _norm64(out, _normal(generator, HIDDEN, std=0.02))
