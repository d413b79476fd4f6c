"""The two forms of the single-GPU decode kernel: a launch of one layer, and a launch of several, which keeps rows that wait in
tensor memory.  A stack must give the bits of its layers launched one by one, with and without the prediction of the next
layer's experts, and with routings whose prediction is always right (eight hot experts) or often wrong."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

SEED = 4321


@pytest.mark.parametrize("predict", [True, False], ids=["predicted", "unpredicted"])
@pytest.mark.parametrize("routing", ["uniform", "hot", "ties"])
def test_a_stack_gives_the_bits_of_its_layers(package, gpu_layers, synth, predict, routing):
    device = torch.device("cuda", 0)
    layers = 12
    provider = package.MoeProvider(layers=layers, max_prefill_tokens=0,
                                   flags=0 if predict else package.provider.FLAG_NO_DECODE_PREDICTION)
    try:
        for layer in range(layers):
            provider.bind_layer(layer, gpu_layers(layer % 3)["cuda"])
        bias = synth.hot_expert_bias(range(3, 256, 32)).to(device) if routing == "hot" else None
        provider.set_router_hooks(bias, quantize_eighths=routing == "ties")
        for n_layers in (1, 2, 3, 7, layers):
            for first in (0, layers - n_layers):
                x = synth.activations(SEED + n_layers, 1, "residual", first)[0].to(device)
                want = x
                for layer in range(first, first + n_layers):
                    want = provider.decode_layer(want, layer)
                got = torch.empty_like(x)
                for _ in range(3):                 # back to back: the exchange words of one launch meet the next
                    provider.decode_stack(x, got, first_layer=first, n_layers=n_layers)
                provider.sync_metrics()
                assert torch.equal(got, want), (n_layers, first)
    finally:
        provider.set_router_hooks(None, quantize_eighths=False)
        provider.release()
