"""The decode producer's wait for an earlier item of its ring (AIMA_MOE_DECODE_IN_FLIGHT): whatever is asked for, the barrier it
looks at must be at most one phase ahead of the item it waits for, because a parity does not show two."""
from __future__ import annotations

import ctypes
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "aima-amd395-qwen36-35b-linux-engine_b200" / "csrc"
SLOTS = 6


def _producer_stands_still(limit: int, items: int = 60) -> bool:
    """The producer's rule on the quickest possible ring: every item has landed and been handed back when the next is issued."""
    landings = [0] * SLOTS                                 # completed phases of full[s]
    landed = 0
    for item in range(items):
        while limit > 0 and item - landed >= limit:
            if landings[landed % SLOTS] & 1 == (landed // SLOTS) & 1:
                return True                                # the phase asked for looks incomplete: nothing will complete it
            landed += 1
        landings[item % SLOTS] += 1
    return False


def test_a_limit_beyond_the_ring_would_stand_still():
    assert not any(_producer_stands_still(limit) for limit in range(SLOTS + 1))
    assert all(_producer_stands_still(limit) for limit in range(SLOTS + 1, 2 * SLOTS + 1))


def test_every_limit_is_held_to_the_ring(tmp_path):
    source = tmp_path / "limit.cu"
    source.write_text('#include "decode_kernel.cuh"\n'
                      'extern "C" __attribute__((visibility("default"))) int limit_for(int asked) { return aima::decode_in_flight_limit(asked); }\n'
                      'extern "C" __attribute__((visibility("default"))) int ring_slots() { return aima::kDecodeRingSlots; }\n')
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    library = tmp_path / "liblimit.so"
    subprocess.run([nvcc, "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", str(CSRC), "-o", str(library), str(source)], check=True)
    probe = ctypes.CDLL(str(library))
    assert probe.ring_slots() == SLOTS
    for asked in (-(2 ** 31), -1, 0, 1, 3, 5, 6, 7, 8, 12, 13, 1000, 2 ** 31 - 1):
        limit = probe.limit_for(asked)
        assert 0 <= limit <= SLOTS and not _producer_stands_still(limit), asked
        if 0 <= asked <= SLOTS:
            assert limit == asked


_CHILD = """
import sys
sys.path.insert(0, {tests!r})
import conftest, torch
package = conftest.load_package()
provider = package.MoeProvider(layers=4, max_prefill_tokens=0)
weights = package.synth.layer_weights_cuda_fast(7, 0, torch.device("cuda", 0))
for layer in range(4):
    provider.bind_layer(layer, weights)
x = package.synth.activations(7, 1, "residual", 0)[0].cuda()
stack, call = torch.empty_like(x), torch.empty_like(x)
provider.decode_stack(x, stack)
call = provider.decode_layer(x, 0)
provider.sync_metrics()
print(stack.view(torch.int16).tolist(), call.view(torch.int16).tolist())
"""


@pytest.mark.gpu
def test_values_beyond_the_ring_change_no_bit(built_library):
    seen = set()
    for value in ("", "0", "1", "7", "11", "-3"):
        child = subprocess.run([sys.executable, "-c", _CHILD.format(tests=str(ROOT / "tests"))], capture_output=True, text=True,
                               env=dict(os.environ, AIMA_MOE_DECODE_IN_FLIGHT=value), timeout=300)
        assert child.returncode == 0, child.stderr[-2000:]
        seen.add(child.stdout)
    assert len(seen) == 1
