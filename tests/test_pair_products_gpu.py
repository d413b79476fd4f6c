"""GPU tests of the two-SM product kernel, the one-launch dispatch plan, the router of a short call and the streamed LM-head
scan at the sizes where they can go wrong: row counts at the edges of the 32-row steps and of the 256-row tiles, the
lowest and highest token count of each router, vocabularies that end inside a copy or leave warps without rows."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

SEED = 4321


@pytest.mark.parametrize("materialised", [False, True])
@pytest.mark.parametrize("edges", [[1, 2, 31, 32, 33, 63, 64, 65], [127, 128, 129, 255, 256, 257, 272, 511, 512, 513, 769]])
def test_expert_row_counts_at_tile_edges(package, gpu_layers, synth, edges, materialised):
    """Forced routing gives experts exactly these row counts.  Every weighted expert row against an FP32 product of the
    same operands with the same rounding points (up to one BF16 step where the order of summation meets a rounding
    boundary: rel 2^-8 of the value, plus what one step of an activation moves the sum by), and the plan exactly."""
    device = torch.device("cuda", 0)
    weights = gpu_layers(0)["cuda"]
    tokens = -(-(sum(edges) + 5) // 8)
    rows = tokens * 8
    ids = torch.full((rows,), 200, dtype=torch.int32)
    at = 0
    for index, count in enumerate(edges):
        ids[at:at + count] = 3 + 7 * index
        at += count
    ids = ids[torch.randperm(rows, generator=torch.Generator().manual_seed(SEED))].reshape(tokens, 8)
    routing = torch.rand(tokens, 8, generator=torch.Generator().manual_seed(SEED + 1)).to(torch.bfloat16)
    h2 = synth.activations(SEED, tokens, "input", 0).to(device)
    resid = synth.activations(SEED, tokens, "residual", 0).to(device)
    flags = package.provider.FLAG_MATERIALIZED_DISPATCH if materialised else 0
    provider = package.MoeProvider(layers=1, max_prefill_tokens=tokens, flags=flags)
    try:
        provider.bind_layer(0, weights)
        provider.set_forced_routing(ids.to(device), routing.to(device))
        views, dbg = provider.make_debug(tokens, prefill=True, with_logits=False, with_slot_rows=True)
        provider.launch_selected_moe(post_attention=h2, residual_hidden=resid, model_layer=0, debug=views)
        provider.sync_metrics()
        got, counts, sorted_rows = dbg["slot_rows"].float(), dbg["expert_counts"].cpu(), dbg["sorted_rows"].cpu()
    finally:
        provider.release()
    flat = ids.reshape(-1)
    assert torch.equal(counts, torch.bincount(flat, minlength=256).to(torch.int32))
    assert torch.equal(sorted_rows.long(), torch.sort(flat, stable=True).indices)
    for expert in torch.unique(flat).tolist():
        where = (flat == expert).nonzero()[:, 0]
        x = h2[(where // 8).to(device)].float()
        gate, up = (x @ weights["expert_gate_up"][expert].float().T).to(torch.bfloat16).float().split(512, dim=1)
        act = (torch.nn.functional.silu(gate).to(torch.bfloat16).float() * up).to(torch.bfloat16).float()
        down = weights["expert_down"][expert].float()
        want = (act @ down.T) * routing.reshape(-1)[where].float().to(device).unsqueeze(1)
        slack = want.abs() * 2.0 ** -8 + 2.0 ** -7 * act.abs().amax() * down.abs().amax() * 4
        assert ((got[where.to(device)] - want).abs() <= slack).all(), (expert, len(where))


@pytest.mark.parametrize("tokens", [1, 7, 127, 128, 129])
@pytest.mark.parametrize("regime", ["uniform", "ties"])
def test_short_call_router_is_bit_exact(package, oracle, gpu_layers, synth, tokens, regime):
    """Both sides of the short-call limit against the oracle: ids (order included), scores and weights."""
    device = torch.device("cuda", 0)
    provider = package.MoeProvider(layers=1, max_prefill_tokens=tokens)
    try:
        provider.bind_layer(0, gpu_layers(0)["cuda"])
        provider.set_router_hooks(None, quantize_eighths=regime == "ties")
        h2 = synth.activations(SEED + tokens, tokens, "input", 0)
        resid = synth.activations(SEED + tokens, tokens, "residual", 0)
        views, dbg = provider.make_debug(tokens, prefill=True, with_logits=False)
        provider.launch_selected_moe(post_attention=h2.to(device), residual_hidden=resid.to(device), model_layer=0, debug=views)
        provider.sync_metrics()
    finally:
        provider.release()
    view = oracle.OracleLayer(gpu_layers(0)["cpu"], router_bias=None, quant_eighths=regime == "ties")
    want = oracle.router_prefill(h2, view)
    assert torch.equal(dbg["topk_ids"].cpu(), want["ids"])
    assert torch.equal(dbg["topk_scores"].cpu(), want["scores"])
    assert torch.equal(dbg["topk_weights"].cpu(), want["weights"])


@pytest.mark.parametrize("shape", [(31, 120, 512), (33, 136, 2048), (255, 8, 64), (257, 512, 2048), (2049, 264, 512), (4097, 2048, 128)])
def test_gemm_at_tile_edges(package, built_library, shape):
    """Rows and columns on either side of the 32-row steps, 128-column halves and 256-row tiles: one BF16 rounding of an
    FP32 sum, 2^-8 relative, plus the rounding of k partial sums."""
    device = torch.device("cuda", 0)
    m, n, k = shape
    generator = torch.Generator(device=device).manual_seed(SEED + m + n + k)
    a = torch.randn(m, k, generator=generator, device=device).to(torch.bfloat16)
    b = (torch.randn(n, k, generator=generator, device=device) * 0.05).to(torch.bfloat16)
    provider = package.MoeProvider(layers=1, max_prefill_tokens=0)
    try:
        got = provider.gemm(a, b)
        provider.sync_metrics()
    finally:
        provider.release()
    want = a.double() @ b.double().T
    slack = want.abs() * 2.0 ** -8 + k * 2.0 ** -23 * (a.double().abs() @ b.double().abs().T)
    assert ((got.double() - want).abs() <= slack).all()


@pytest.mark.parametrize("rows", [1, 3, 5, 33, 3551, 3553, 7105])
def test_lm_head_rows_at_the_ends_of_copies_and_runs(package, oracle, rows):
    """One row; a last copy of one, three or four rows; just below and above two rows for each of 148 x 12 warps."""
    generator = torch.Generator().manual_seed(SEED + rows)
    weight = (torch.randn(rows, 2048, generator=generator) * 0.02).to(torch.bfloat16)
    hidden = torch.randn(2048, generator=generator).to(torch.bfloat16)
    q, scales, residual = oracle.lm_head_quantize(weight)
    want = oracle.lm_head_certify(weight, q, scales, residual, hidden)
    head = package.LmHead(weight.to("cuda"))
    try:
        for _ in range(2):          # the state of a launch is reset by the next
            logits = head.launch(hidden.to("cuda"))
            result = head.result()
            assert result.hidden_l2 == want["hidden_l2"]
            assert result.maximum_lower_bound == want["maximum_lower_bound"]
            assert result.candidate_count == want["candidate_count"] and result.overflow == 0
            assert result.exact_top1_token_id == want["top1_token"]
            assert result.exact_top1_logit == want["top1_logit"]
            assert torch.equal(logits.cpu(), want["logits"])
    finally:
        head.release()


@pytest.mark.parametrize("flag", [None, "FLAG_MATERIALIZED_DISPATCH", "FLAG_EXACT_ROUTER"])
def test_nan_logits_of_a_short_call_stay_in_their_row(package, oracle, gpu_layers, synth, flag):
    """After a longer call on the same handle: a row of NaN gets the eight lowest experts (all its logits count as -inf) and
    leaves its neighbours' bits alone; a router row with a NaN, one logit of every token, is as good as -inf there."""
    device = torch.device("cuda", 0)
    weights = gpu_layers(0)["cuda"]
    broken = dict(weights, router=weights["router"].clone())
    broken["router"][77, 5] = float("nan")
    tokens, bad, longer = 40, 7, 300
    h2 = synth.activations(SEED, longer, "input", 0).to(device)
    resid = synth.activations(SEED, longer, "residual", 0).to(device)
    with_nan = h2[:tokens].clone()
    with_nan[bad] = float("nan")
    provider = package.MoeProvider(layers=2, max_prefill_tokens=longer, flags=getattr(package.provider, flag) if flag else 0)
    try:
        provider.bind_layer(0, weights)
        provider.bind_layer(1, broken)

        def call(x, layer=0):
            views, dbg = provider.make_debug(len(x), prefill=True, with_logits=False)
            out = provider.launch_selected_moe(post_attention=x, residual_hidden=resid[:len(x)], model_layer=layer, debug=views)
            provider.sync_metrics()
            return out, dbg

        clean, clean_dbg = call(h2[:tokens])
        call(h2)
        got, dbg = call(with_nan)
        others = [t for t in range(tokens) if t != bad]
        assert torch.equal(got[others], clean[others])
        assert torch.equal(dbg["topk_ids"][others], clean_dbg["topk_ids"][others])
        assert sorted(dbg["topk_ids"][bad].tolist()) == list(range(8))      # (the fixed network permutes equal scores)
        assert torch.isnan(got[bad]).all()
        assert int(dbg["expert_offsets"][256]) == tokens * 8
        assert torch.equal(dbg["sorted_rows"].sort().values.cpu(), torch.arange(tokens * 8, dtype=torch.int32))
        call(h2)
        _, dbg = call(h2[:tokens], layer=1)
    finally:
        provider.release()
    bias = torch.zeros(256)
    bias[77] = float("-inf")
    want = oracle.router_prefill(h2[:tokens].cpu(), oracle.OracleLayer(gpu_layers(0)["cpu"], router_bias=bias))
    assert torch.equal(dbg["topk_ids"].cpu(), want["ids"])
    assert torch.equal(dbg["topk_scores"].cpu(), want["scores"])
    assert torch.equal(dbg["topk_weights"].cpu(), want["weights"])


@pytest.mark.parametrize("flag", [None, "FLAG_EXACT_ROUTER", "FLAG_AUDIT_ROUTER"])
def test_nan_logit_of_a_long_call_counts_as_minus_infinity(package, oracle, gpu_layers, synth, flag):
    """The certified router beyond the short calls: one NaN logit in every token neither takes a slot nor costs one."""
    device = torch.device("cuda", 0)
    weights = gpu_layers(0)["cuda"]
    broken = dict(weights, router=weights["router"].clone())
    broken["router"][77, 5] = float("nan")
    tokens = 200
    h2 = synth.activations(SEED + 3, tokens, "input", 0)
    provider = package.MoeProvider(layers=1, max_prefill_tokens=tokens, flags=getattr(package.provider, flag) if flag else 0)
    try:
        provider.bind_layer(0, broken)
        views, dbg = provider.make_debug(tokens, prefill=True, with_logits=False)
        provider.launch_selected_moe(post_attention=h2.to(device), residual_hidden=h2.to(device), model_layer=0, debug=views)
        metrics = provider.sync_metrics()
    finally:
        provider.release()
    bias = torch.zeros(256)
    bias[77] = float("-inf")
    want = oracle.router_prefill(h2, oracle.OracleLayer(gpu_layers(0)["cpu"], router_bias=bias))
    assert torch.equal(dbg["topk_ids"].cpu(), want["ids"])
    assert torch.equal(dbg["topk_scores"].cpu(), want["scores"])
    assert torch.equal(dbg["topk_weights"].cpu(), want["weights"])
    assert metrics.router_audit_mismatches == 0 and metrics.router_bound_violations == 0


def test_calls_that_do_not_filter_leave_the_filter_statistics_alone(package, gpu_layers, synth):
    device = torch.device("cuda", 0)
    provider = package.MoeProvider(layers=1, max_prefill_tokens=129)
    try:
        provider.bind_layer(0, gpu_layers(0)["cuda"])
        h2 = synth.activations(SEED, 129, "input", 0).to(device)
        seen = []
        for tokens in (129, 128, 1):
            provider.launch_selected_moe(post_attention=h2[:tokens], residual_hidden=h2[:tokens], model_layer=0)
            metrics = provider.sync_metrics()
            seen.append((metrics.router_tokens, metrics.router_candidates))
        assert seen[0][0] == 129 and 8 * 129 <= seen[0][1] <= 64 * 129
        assert seen[1:] == seen[:1] * 2
    finally:
        provider.release()


@pytest.mark.parametrize("tokens", [1025, 1100, 3584, 3585])
def test_copied_and_gathered_tiles_give_the_same_bits(package, gpu_layers, synth, tokens):
    """Calls in which some tiles are copied into expert order and others gathered by token: row counts on both sides of the
    crossing (96) and of its halves and doubles, against the form that copies everything."""
    device = torch.device("cuda", 0)
    edges = [1, 31, 33, 64, 95, 96, 97, 128, 160, 161, 192, 193, 256, 257, 320, 321, 353, 449, 513, 577]
    rows = tokens * 8
    ids = torch.full((rows,), 200, dtype=torch.int32)
    at = 0
    for index, count in enumerate(edges):
        ids[at:at + count] = 3 + 7 * index
        at += count
    generator = torch.Generator().manual_seed(SEED + tokens)
    ids = ids[torch.randperm(rows, generator=generator)].reshape(tokens, 8).to(device)
    routing = torch.rand(tokens, 8, generator=generator).to(torch.bfloat16).to(device)
    h2 = synth.activations(SEED, tokens, "input", 0).to(device)
    resid = synth.activations(SEED, tokens, "residual", 0).to(device)
    results = []
    for flags in (0, package.provider.FLAG_MATERIALIZED_DISPATCH):
        provider = package.MoeProvider(layers=1, max_prefill_tokens=tokens, flags=flags)
        try:
            provider.bind_layer(0, gpu_layers(0)["cuda"])
            provider.set_forced_routing(ids, routing)
            views, dbg = provider.make_debug(tokens, prefill=True, with_logits=False, with_slot_rows=True)
            out = provider.launch_selected_moe(post_attention=h2, residual_hidden=resid, model_layer=0, debug=views)
            provider.sync_metrics()
            results.append((out, dbg["slot_rows"], dbg["shared_scaled"]))
        finally:
            provider.release()
    for mixed, copied in zip(*results):
        assert torch.equal(mixed, copied)
