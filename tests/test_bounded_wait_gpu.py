"""GPU test of the bounded wait that whole warps take: completed before the limit, never completed, and completed about
when the limit runs out, all 32 lanes get the same verdict and the kernel ends."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "aima-amd395-qwen36-35b-linux-engine_b200" / "csrc"
BLOCKS = 592


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    library = tmp_path_factory.mktemp("wait") / "libbounded_wait_probe.so"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-O3", "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", str(CSRC), "-o", str(library), str(ROOT / "tests" / "bounded_wait_probe.cu")], check=True)
    run = ctypes.CDLL(str(library)).run_wait_probe
    run.argtypes = [ctypes.c_void_p, ctypes.c_uint64, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]

    def call(delays_ns: torch.Tensor, limit_ns: int):
        verdicts = torch.full((BLOCKS, 32), -1, dtype=torch.int32, device="cuda")
        flags = torch.full((BLOCKS,), -1, dtype=torch.int32, device="cuda")
        delays_ns = delays_ns.to("cuda")
        torch.cuda.synchronize()
        assert run(delays_ns.data_ptr(), limit_ns, BLOCKS, verdicts.data_ptr(), flags.data_ptr()) == 0
        return verdicts.cpu(), flags.cpu()

    return call


@pytest.mark.parametrize("limit_ns", [0, 20_000, 200_000])
def test_all_lanes_get_one_verdict(probe, limit_ns):
    never = torch.arange(BLOCKS) % 4 == 0
    at_once = torch.arange(BLOCKS) % 4 == 1
    for repeat in range(8):
        # the others complete within 25 us of the limit, on both sides of it
        delays = limit_ns + torch.randint(-25_000, 25_000, (BLOCKS,), generator=torch.Generator().manual_seed(repeat))
        delays = delays.clamp(min=0).masked_fill(never, -1).masked_fill(at_once, 0)
        verdicts, flags = probe(delays, limit_ns)
        assert torch.equal(verdicts, verdicts[:, :1].expand_as(verdicts))
        assert (verdicts[never] == 0).all()
        if limit_ns > 0:
            assert (verdicts[at_once] == 1).all()
        assert torch.equal(flags != 0, verdicts[:, 0] == 0)
