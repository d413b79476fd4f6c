"""GPU test of the two-SM kernel's accumulators, which the epilogue warps of both blocks hand back to the block that issues the
products: with one K stage per unit and many units per pair of blocks, each accumulator is overwritten as soon as it is handed
back.  Operands of -1, 0 and 1 make every result exact, so a value read late shows as a wrong bit."""
from __future__ import annotations

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(8192, 4096, 64), (8191, 4088, 64), (4097, 8192, 128)])
def test_accumulators_are_read_before_they_are_overwritten(product_probe, m, n, k):
    generator = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = [torch.randint(-1, 2, (m, k), generator=generator, device="cuda").to(torch.bfloat16) for _ in range(2)]
    b = torch.randint(-1, 2, (n, k), generator=generator, device="cuda").to(torch.bfloat16)
    want = [(x.float() @ b.float().T).to(torch.bfloat16) for x in a]           # |sum| <= 128: exact in BF16
    out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for index in range(40):
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        pointers = [ctypes.c_void_p(t.data_ptr()) for t in (a[index & 1], b, out)]
        assert product_probe.run_dense(*pointers, m, n, k, sms, ctypes.c_void_p(status.data_ptr()), ctypes.c_uint64(2_000_000_000)) == 0
        torch.cuda.synchronize()
        wrong += (out != want[index & 1]).sum()
    assert status.item() == 0
    assert int(wrong) == 0
