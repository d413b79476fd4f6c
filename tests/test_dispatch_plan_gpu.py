"""The dispatch plan from counts per chunk of rows, and the router forms that leave those counts: a token's dots shared by
four, two or one warps, logits from four or two runs of K.  Routing is compared with the router that computes all 256
canonical logits (which counts its rows in a kernel of its own), the plan with a stable sort of the ids on the CPU."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

SEED = 8642
CAPACITY = 4111


@pytest.fixture(scope="module")
def provider(package, gpu_layers):
    provider = package.MoeProvider(layers=1, max_prefill_tokens=CAPACITY)
    provider.bind_layer(0, gpu_layers(0)["cuda"])
    yield provider
    provider.release()


def _run(provider, h2, exact: bool):
    views, tensors = provider.make_debug(h2.shape[0], prefill=True, with_logits=exact)
    out = provider.launch_selected_moe(post_attention=h2, residual_hidden=torch.zeros_like(h2), model_layer=0, debug=views)
    metrics = provider.sync_metrics()
    return out, {k: v.cpu() for k, v in tensors.items()}, metrics


def _check_plan(dbg, metrics):
    flat = dbg["topk_ids"].reshape(-1).long()
    counts = torch.bincount(flat, minlength=256)
    assert torch.equal(dbg["expert_counts"].long(), counts)
    assert torch.equal(dbg["expert_offsets"].long(), torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]))
    assert torch.equal(dbg["sorted_rows"].long(), torch.sort(flat, stable=True).indices)
    assert metrics.last_padded_routed_rows == int(((counts + 31) // 32 * 32).sum())


# both sides of every limit on 148 SMs: 128 (all logits canonical), 592 and 1184 (warps per token), 1024 (runs of K), and
# odd counts whose last chunk, tile and block of the plan are ragged
@pytest.mark.parametrize("tokens", [1, 9, 128, 129, 255, 592, 593, 1024, 1025, 1184, 1185, 2047, CAPACITY])
@pytest.mark.parametrize("routing", ["uniform", "hot", "ties"])
def test_routing_and_plan_at_the_limits_of_the_router_forms(provider, synth, tokens, routing):
    device = torch.device("cuda", 0)
    h2 = torch.randn(tokens, 2048, generator=torch.Generator().manual_seed(SEED + tokens)).to(torch.bfloat16).to(device)
    bias = synth.hot_expert_bias(range(3, 256, 32)).to(device) if routing == "hot" else None
    provider.set_router_hooks(bias, quantize_eighths=routing == "ties")
    try:
        out, got, metrics = _run(provider, h2, exact=False)
        _check_plan(got, metrics)
        want_out, want, metrics = _run(provider, h2, exact=True)
        _check_plan(want, metrics)
    finally:
        provider.set_router_hooks(None, quantize_eighths=False)
    for name in ("topk_ids", "topk_scores", "topk_weights", "sorted_rows"):
        assert torch.equal(got[name], want[name]), name
    assert torch.equal(out, want_out)             # same rows, same weights, same products


@pytest.mark.parametrize("tokens", [1, 130, 1025])
def test_plan_of_forced_ids_with_repeats(provider, tokens):
    """Ids that no router gives: an expert several times in a token, one expert for all rows of a chunk."""
    device = torch.device("cuda", 0)
    generator = torch.Generator().manual_seed(SEED)
    ids = torch.randint(0, 4, (tokens, 8), generator=generator, dtype=torch.int32) * 85
    ids[: tokens // 2] = 255
    h2 = torch.randn(tokens, 2048, generator=generator).to(torch.bfloat16).to(device)
    provider.set_forced_routing(ids.to(device), torch.full((tokens, 8), 0.125, dtype=torch.bfloat16, device=device))
    try:
        _, got, metrics = _run(provider, h2, exact=False)
    finally:
        provider.set_forced_routing(None, None)
    assert torch.equal(got["topk_ids"], ids)
    _check_plan(got, metrics)
