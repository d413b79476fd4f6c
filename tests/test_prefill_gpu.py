"""GPU parity of the prefill path through the C ABI: routing bit-exact against the CPU oracle
(ids with the reference's tie order, scores, weights), the dispatch plan exact, layer outputs
within the stated BF16 tolerance, and agreement with the committed torch golden vectors."""
from __future__ import annotations

from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SEED = 1234
MAX_ABS = 2.0e-2      # BASELINE north_star tolerance on the MoE output (routed + shared)
COSINE = 0.9999
GOLDEN = Path(__file__).resolve().parent / "golden"


@pytest.fixture(scope="module")
def provider(package, gpu_layers):
    provider = package.MoeProvider(layers=2, max_prefill_tokens=1024)
    for layer in range(2):
        provider.bind_layer(layer, gpu_layers(layer)["cuda"])
    yield provider
    provider.release()


def _cosine(a, b):
    a, b = a.double().reshape(-1), b.double().reshape(-1)
    return float((a @ b) / (a.norm() * b.norm()).clamp_min(1e-30))


def _run(provider, layer, h2, resid):
    device = torch.device("cuda", 0)
    tokens = h2.shape[0]
    views, tensors = provider.make_debug(tokens, prefill=True)
    out = provider.launch_selected_moe(post_attention=h2.to(device), residual_hidden=resid.to(device),
                                       model_layer=layer, debug=views)
    metrics = provider.sync_metrics()
    return out.cpu(), {k: v.cpu() for k, v in tensors.items()}, metrics


def _check_against_oracle(oracle, layer_view, h2, resid, out, dbg, metrics, select=None):
    tokens = h2.shape[0]
    routing = oracle.router_prefill(h2, layer_view)
    assert torch.equal(dbg["router_logits"], routing["logits"])
    assert torch.equal(dbg["topk_ids"], routing["ids"])                 # order included
    assert torch.equal(dbg["topk_scores"], routing["scores"])
    assert torch.equal(dbg["topk_weights"], routing["weights"])
    plan = oracle.dispatch_plan(routing["ids"])
    assert torch.equal(dbg["expert_counts"], plan["counts"])
    assert torch.equal(dbg["expert_offsets"], plan["offsets"])
    assert torch.equal(dbg["sorted_rows"], plan["sorted_rows"])
    assert metrics.last_padded_routed_rows == plan["padded_rows"]
    rows = list(range(tokens)) if select is None else select
    want = oracle.prefill_layer(h2, resid, layer_view, select=rows)
    got_moe = dbg["routed"][rows].float() + dbg["shared_scaled"][rows].float()
    want_moe = want["routed"].float() + want["shared_scaled"].float()
    assert torch.isfinite(out.float()).all()
    assert (got_moe - want_moe).abs().max() <= MAX_ABS
    assert _cosine(got_moe, want_moe) >= COSINE
    assert _cosine(dbg["shared_scaled"][rows], want["shared_scaled"]) >= COSINE
    assert _cosine(dbg["routed"][rows], want["routed"]) >= COSINE
    # final hidden = bf16(residual + bf16(routed + shared)) from the GPU's own stage outputs
    combined = (dbg["routed"].float() + dbg["shared_scaled"].float()).to(torch.bfloat16)
    assert torch.equal(out, (resid.float() + combined.float()).to(torch.bfloat16))
    ulp = want["out"].float().abs() * 2.0 ** -7
    assert ((out[rows].float() - want["out"].float()).abs() <= ulp + MAX_ABS).all()


@pytest.mark.parametrize("tokens", [1, 7, 16, 33, 257])
def test_prefill_layer_matches_oracle(provider, oracle, gpu_layers, synth, tokens):
    layer = tokens % 2
    h2 = synth.activations(SEED + tokens, tokens, "input", layer)
    resid = synth.activations(SEED + tokens, tokens, "residual", layer)
    out, dbg, metrics = _run(provider, layer, h2, resid)
    select = None if tokens <= 33 else list(range(0, tokens, 16)) + [tokens - 1]
    _check_against_oracle(oracle, gpu_layers(layer)["oracle"], h2, resid, out, dbg, metrics, select)


def test_prefill_tie_stress_routing_is_bit_exact(provider, oracle, gpu_layers, synth):
    """Router logits rounded to multiples of 1/8: many exact ties, ids must keep the reference's
    order (BASELINE config 4c)."""
    tokens = 512
    provider.set_router_hooks(None, quantize_eighths=True)
    try:
        h2 = synth.activations(SEED + 900, tokens, "input", 0)
        resid = synth.activations(SEED + 900, tokens, "residual", 0)
        out, dbg, metrics = _run(provider, 0, h2, resid)
        tied = oracle.OracleLayer(gpu_layers(0)["cpu"], quant_eighths=True)
        routing = oracle.router_prefill(h2, tied)
        assert torch.equal(dbg["topk_ids"], routing["ids"])
        assert torch.equal(dbg["topk_weights"], routing["weights"])
        scores = routing["scores"]
        assert int((scores[:, :-1] == scores[:, 1:]).sum()) > tokens      # ties are everywhere
        _check_against_oracle(oracle, tied, h2, resid, out, dbg, metrics, select=[0, 100, 511])
    finally:
        provider.set_router_hooks(None, quantize_eighths=False)


def test_prefill_hot_and_skewed_routing(provider, oracle, gpu_layers, synth):
    device = torch.device("cuda", 0)
    tokens = 300
    h2 = synth.activations(SEED + 901, tokens, "input", 1)
    resid = synth.activations(SEED + 901, tokens, "residual", 1)
    hot = [0, 31, 32, 100, 101, 200, 254, 255]
    for bias in (synth.hot_expert_bias(hot), synth.zipf_router_bias(SEED)):
        provider.set_router_hooks(bias.to(device), quantize_eighths=False)
        try:
            out, dbg, metrics = _run(provider, 1, h2, resid)
            view = oracle.OracleLayer(gpu_layers(1)["cpu"], router_bias=bias)
            _check_against_oracle(oracle, view, h2, resid, out, dbg, metrics, select=[0, 1, 150, 299])
        finally:
            provider.set_router_hooks(None, quantize_eighths=False)
    # hot case: exactly eight populated experts, 248 empty ones
    provider.set_router_hooks(synth.hot_expert_bias(hot).to(device), quantize_eighths=False)
    try:
        _, dbg, _ = _run(provider, 1, h2, resid)
        counts = dbg["expert_counts"]
        assert counts[hot].tolist() == [tokens] * 8 and int(counts.sum()) == tokens * 8
    finally:
        provider.set_router_hooks(None, quantize_eighths=False)


def _run_production(provider, layer, h2, resid):
    """Same call without the logits view: the production (certified, tensor-core filtered) router."""
    device = torch.device("cuda", 0)
    views, tensors = provider.make_debug(h2.shape[0], prefill=True, with_logits=False)
    out = provider.launch_selected_moe(post_attention=h2.to(device), residual_hidden=resid.to(device),
                                       model_layer=layer, debug=views)
    metrics = provider.sync_metrics()
    return out.cpu(), {k: v.cpu() for k, v in tensors.items()}, metrics


@pytest.mark.parametrize("regime", ["uniform", "ties", "hot", "zipf"])
def test_certified_router_is_bit_exact(provider, oracle, gpu_layers, synth, regime):
    """The production router filters candidates with tensor-core logits and recomputes only those
    with the canonical dot; ids (order included), scores and weights must equal the oracle's."""
    device = torch.device("cuda", 0)
    tokens = 700
    layer = 1
    bias, quant = None, False
    if regime == "ties":
        quant = True
    elif regime == "hot":
        bias = synth.hot_expert_bias([5, 6, 7, 64, 65, 128, 200, 255])
    elif regime == "zipf":
        bias = synth.zipf_router_bias(SEED + 3)
    provider.set_router_hooks(None if bias is None else bias.to(device), quantize_eighths=quant)
    try:
        h2 = synth.activations(SEED + 950, tokens, "input", layer)
        resid = synth.activations(SEED + 950, tokens, "residual", layer)
        before = provider.sync_metrics()
        out, dbg, metrics = _run_production(provider, layer, h2, resid)
        view = oracle.OracleLayer(gpu_layers(layer)["cpu"], router_bias=bias, quant_eighths=quant)
        routing = oracle.router_prefill(h2, view)
        assert torch.equal(dbg["topk_ids"], routing["ids"])
        assert torch.equal(dbg["topk_scores"], routing["scores"])
        assert torch.equal(dbg["topk_weights"], routing["weights"])
        routed_tokens = metrics.router_tokens - before.router_tokens
        candidates = metrics.router_candidates - before.router_candidates
        assert routed_tokens == tokens
        assert 8 * tokens <= candidates <= 64 * tokens          # a filter, not a full recomputation
        # and the exact router gives the same layer output bits (same routing, same products)
        out_exact, dbg_exact, _ = _run(provider, layer, h2, resid)
        assert torch.equal(out, out_exact)
        assert torch.equal(dbg["shared_scaled"], dbg_exact["shared_scaled"])
    finally:
        provider.set_router_hooks(None, quantize_eighths=False)


@pytest.mark.parametrize("tokens", [1, 16])
def test_prefill_matches_torch_golden(provider, gpu_layers, synth, tokens):
    """BASELINE config 0 against the committed torch-CPU vectors (tests/golden/make_golden.py)."""
    data = np.load(GOLDEN / f"config0_T{tokens}.npz")
    seed, layer, _ = (int(v) for v in data["seed"])
    assert seed == SEED and layer == 0
    h2 = synth.activations(seed, tokens, "input", layer)
    resid = synth.activations(seed, tokens, "residual", layer)
    out, dbg, _ = _run(provider, layer, h2, resid)

    def bf16(bits):
        return torch.from_numpy(bits.view(np.int16).copy()).view(torch.bfloat16)

    golden_sets = torch.from_numpy(data["topk_indices"]).sort(dim=-1).values
    same = (dbg["topk_ids"].long().sort(dim=-1).values == golden_sets).all(dim=-1)
    assert same.float().mean() >= 0.9
    rows = same.nonzero().reshape(-1)
    golden_moe = bf16(data["moe_out"]).float() + bf16(data["shared_out"]).float()
    got_moe = dbg["routed"].float() + dbg["shared_scaled"].float()
    assert (got_moe[rows] - golden_moe[rows]).abs().max() <= MAX_ABS
    assert _cosine(got_moe[rows], golden_moe[rows]) >= COSINE


def test_prefill_stack_matches_chained_layers(provider, oracle, gpu_layers, synth):
    """Two layers through the stack entry point equal norm + single-layer calls chained by hand."""
    device = torch.device("cuda", 0)
    tokens = 64
    x = synth.activations(SEED + 902, tokens, "residual", 0).to(device)
    y = torch.empty_like(x)
    provider.prefill_stack(x, y, first_layer=0, n_layers=2)
    current = x
    for layer in range(2):
        _, h2 = provider.rmsnorm(current, gpu_layers(layer)["cuda"]["post_attention_layernorm"])
        current = provider.launch_selected_moe(post_attention=h2, residual_hidden=current, model_layer=layer)
    provider.sync_metrics()
    assert torch.equal(y.cpu(), current.cpu())
    # teacher-forced check of layer 0 against the oracle
    _, h2 = provider.rmsnorm(x, gpu_layers(0)["cuda"]["post_attention_layernorm"])
    _, h2_cpu = oracle.rmsnorm(x.cpu(), gpu_layers(0)["cpu"]["post_attention_layernorm"])
    assert torch.equal(h2.cpu(), h2_cpu)


def test_fused_boundary_equals_the_separate_calls(provider, oracle, gpu_layers, synth):
    """attn_out + residual -> norm -> MoE -> next layer's norm in one call: same bits as the three calls."""
    device = torch.device("cuda", 0)
    tokens = 96
    attn_out = synth.activations(SEED + 910, tokens, "input", 0).to(device)
    residual_in = synth.activations(SEED + 910, tokens, "residual", 0).to(device)
    norm0 = gpu_layers(0)["cuda"]["post_attention_layernorm"]
    norm1 = gpu_layers(1)["cuda"]["post_attention_layernorm"]
    layer_out, next_norm = provider.prefill_fused(attn_out, residual_in, 0, next_norm_weight=norm1)
    after_attn, h2 = provider.rmsnorm(attn_out, norm0, residual=residual_in)
    want = provider.launch_selected_moe(post_attention=h2, residual_hidden=after_attn, model_layer=0)
    _, want_next = provider.rmsnorm(want, norm1)
    provider.sync_metrics()
    assert torch.equal(layer_out, want)
    assert torch.equal(next_norm, want_next)
    # the fused exit norm against the CPU oracle's norm of the same rows
    _, oracle_next = oracle.rmsnorm(layer_out.cpu(), gpu_layers(1)["cpu"]["post_attention_layernorm"])
    assert torch.equal(next_norm.cpu(), oracle_next)
    # and the entry (add + norm) against the oracle
    oracle_after, oracle_h2 = oracle.rmsnorm(attn_out.cpu(), gpu_layers(0)["cpu"]["post_attention_layernorm"],
                                             residual=residual_in.cpu())
    assert torch.equal(after_attn.cpu(), oracle_after)
    assert torch.equal(h2.cpu(), oracle_h2)
    only_out, none = provider.prefill_fused(attn_out, residual_in, 0)
    provider.sync_metrics()
    assert none is None and torch.equal(only_out, want)


def test_prefill_argument_checks(provider, package, synth):
    device = torch.device("cuda", 0)
    h2 = synth.activations(1, 4).to(device)
    with pytest.raises(package.AimaMoeError) as alias:
        provider.launch_selected_moe(post_attention=h2, residual_hidden=h2.clone(), model_layer=0, out=h2)
    assert alias.value.status == -4
    big = torch.zeros(2048, 2048, dtype=torch.bfloat16, device=device)
    with pytest.raises(package.AimaMoeError) as capacity:
        provider.launch_selected_moe(post_attention=big, residual_hidden=big.clone(), model_layer=0)
    assert capacity.value.status == -8


@pytest.mark.parametrize("tokens", [40, 300])
@pytest.mark.parametrize("flag", [None, "FLAG_EXACT_ROUTER", "FLAG_SIMT_PRODUCTS"])
def test_misaligned_pointers_are_refused_before_any_launch(package, gpu_layers, synth, tokens, flag):
    """A view that starts two bytes into its allocation, as input or output: an error from the host, whatever kernel would
    have met it first, and the handle goes on working."""
    device = torch.device("cuda", 0)
    good = synth.activations(SEED, tokens, "input", 0).to(device)
    shifted = torch.empty(tokens * 2048 + 8, dtype=torch.bfloat16, device=device)[1:1 + tokens * 2048].view(tokens, 2048)
    shifted.copy_(good)
    provider = package.MoeProvider(layers=1, max_prefill_tokens=tokens, flags=getattr(package.provider, flag) if flag else 0)
    try:
        provider.bind_layer(0, gpu_layers(0)["cuda"])
        want = provider.launch_selected_moe(post_attention=good, residual_hidden=good, model_layer=0)
        provider.sync_metrics()
        calls = [lambda: provider.launch_selected_moe(post_attention=shifted, residual_hidden=good, model_layer=0),
                 lambda: provider.launch_selected_moe(post_attention=good, residual_hidden=shifted, model_layer=0),
                 lambda: provider.launch_selected_moe(post_attention=good, residual_hidden=good, model_layer=0, out=shifted),
                 lambda: provider.prefill_stack(shifted, torch.empty_like(good)),
                 lambda: provider.prefill_stack(good, shifted),
                 lambda: provider.gemm(shifted, good)]
        for call in calls:
            launched = provider.sync_metrics().kernel_launches
            with pytest.raises(package.AimaMoeError) as error:
                call()
            assert error.value.status == -1                                # AIMA_MOE_ERR_INVALID_ARGUMENT
            assert provider.sync_metrics().kernel_launches == launched
        got = provider.launch_selected_moe(post_attention=good, residual_hidden=good, model_layer=0)
        provider.sync_metrics()
        assert torch.equal(got, want)
    finally:
        provider.release()
