"""GPU test of what the product kernels do when a wait runs out: with a limit shorter than a unit takes, the two-SM one stops
in both blocks of every pair, the one-SM one in its block; copies and MMAs land, it returns with a status, and the next launch
gives the right bits."""
from __future__ import annotations

import ctypes
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

NO_LIMIT = 2_000_000_000


def _p(tensor: torch.Tensor) -> ctypes.c_void_p:
    return ctypes.c_void_p(tensor.data_ptr())


def _check(launch, out: torch.Tensor, limit_ns: int, must_run_out: bool) -> None:
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(limit: int) -> int:
        status.zero_()
        torch.cuda.synchronize()
        assert launch(status, ctypes.c_uint64(limit)) == 0
        torch.cuda.synchronize()
        return int(status.item())

    out.zero_()
    assert run(NO_LIMIT) == 0
    want = out.clone()
    for _ in range(10):
        out.zero_()
        started = time.perf_counter()
        ran_out = run(limit_ns) != 0
        assert time.perf_counter() - started < 8.0        # the drain's own limit is 2 s for the MMAs and 2 s for the copies
        assert ran_out or (torch.equal(out, want) and not must_run_out)
        out.zero_()
        assert run(NO_LIMIT) == 0
        assert torch.equal(out, want)


@pytest.mark.parametrize("limit_ns", [0, 6_000, 20_000, 5_000_000])
def test_dense_product_stops_and_recovers(product_probe, limit_ns):
    m, n, k = 4096, 2048, 8192         # a unit is 128 stages, more than 30 us
    generator = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(m, k, generator=generator, device="cuda").to(torch.bfloat16)
    b = torch.randn(n, k, generator=generator, device="cuda").to(torch.bfloat16)
    out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _check(lambda status, limit: product_probe.run_dense(_p(a), _p(b), _p(out), m, n, k, sms, _p(status), limit), out, limit_ns,
           must_run_out=limit_ns <= 20_000)


@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("limit_ns", [0, 4_000, 12_000, 5_000_000])
def test_gathered_product_stops_and_recovers(product_probe, limit_ns, pair):
    tokens, experts = 1024, 24
    generator = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(tokens, 2048, generator=generator, device="cuda").to(torch.bfloat16)
    weights = (torch.randn(experts, 1024, 2048, generator=generator, device="cuda") * 0.05).to(torch.bfloat16)
    heights = [256, 160, 33, 96, 1, 224, 31, 128]
    tiles = [(e, min(heights[(3 * e + t) % len(heights)], 256 if pair else 128)) for e in range(experts) for t in range(4)]
    rows = torch.tensor([r for _, r in tiles], dtype=torch.int32)
    total = int(rows.sum())
    row0 = (rows.cumsum(0) - rows).to(torch.int32).cuda()
    tile_expert = torch.tensor([e for e, _ in tiles], dtype=torch.int32).cuda()
    rows = rows.cuda()
    count = torch.tensor([len(tiles)], dtype=torch.int32, device="cuda")
    sorted_rows = torch.randint(0, tokens * 8, (total,), generator=torch.Generator().manual_seed(5), dtype=torch.int32).cuda()
    out = torch.empty(total, 512, dtype=torch.bfloat16, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    operands = product_probe.operands(x=x, gate_up=weights, tile_expert=tile_expert, tile_row0=row0, tile_rows=rows,
                                      tile_count=count, sorted_rows=sorted_rows, act=out, tokens=tokens, rows=total,
                                      experts=experts, max_tiles=len(tiles))
    _check(lambda status, limit: product_probe.run_gate_up(ctypes.byref(operands), pair, 0, sms, _p(status), limit),
           out, limit_ns, must_run_out=limit_ns == 0 and pair == 1)
