"""GPU tests of the two ways the gate_up product takes its rows by token index, TMA gathers and cp.async: both give the bits of
the one-SM kernel with the shared expert's tiles in the launch and without, at the edges of the 32-row steps and of the 256-row
tiles; both stop when a wait runs out and leave a device on which the next launch is right; and the calls on either side of the
limit between them give the bits of a copy in expert order."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest
import torch

from test_product_limit_gpu import _check

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
SEED = 987
LIMIT = ctypes.c_uint64(2_000_000_000)
TOKENS, EXPERTS = 1029, 24
HEIGHTS = [256, 1, 31, 32, 33, 64, 95, 127, 128, 129, 160, 161, 224, 225, 255]


@pytest.fixture(scope="module")
def feed_probe(tmp_path_factory):
    library = tmp_path_factory.mktemp("feed") / "librow_feed_probe.so"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-O3", "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", str(ROOT / "aima-amd395-qwen36-35b-linux-engine_b200" / "csrc"), "-o", str(library),
                    str(ROOT / "tests" / "row_feed_probe.cu")], check=True)
    return ctypes.CDLL(str(library))


def _normal(seed: int, *shape: int, std: float = 1.0) -> torch.Tensor:
    generator = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=generator, device="cuda") * std).to(torch.bfloat16)


@pytest.fixture(scope="module")
def problem():
    """Rows of 24 experts, several ragged tiles each; every token index at least once, the last token's row included."""
    tall = [(e, HEIGHTS[(4 * e + t) % len(HEIGHTS)]) for e in range(EXPERTS) for t in range(4)]
    total = sum(rows for _, rows in tall)
    generator = torch.Generator().manual_seed(SEED)
    flat = torch.cat([torch.randperm(TOKENS * 8, generator=generator) for _ in range(-(-total // (TOKENS * 8)))])[:total]
    return {
        "x": _normal(SEED, TOKENS, 2048), "gate_up": _normal(SEED + 1, EXPERTS, 1024, 2048, std=0.05),
        "shared_gate": _normal(SEED + 2, 512, 2048, std=0.05), "shared_up": _normal(SEED + 3, 512, 2048, std=0.05),
        "sorted_rows": flat.to(torch.int32).cuda(), "tall": tall, "total": total,
        "sms": torch.cuda.get_device_properties(0).multi_processor_count,
    }


def _plan(tall, cap: int) -> dict:
    tiles, at = [], 0
    for expert, rows in tall:
        tiles += [(expert, at + low, min(cap, rows - low)) for low in range(0, rows, cap)]
        at += rows
    columns = [torch.tensor(column, dtype=torch.int32, device="cuda") for column in zip(*tiles)]
    return {"tile_expert": columns[0], "tile_row0": columns[1], "tile_rows": columns[2],
            "tile_count": torch.tensor([len(tiles)], dtype=torch.int32, device="cuda"), "max_tiles": len(tiles)}


def _operands(product_probe, problem, cap: int, **changed):
    values = {name: problem[name] for name in ("x", "gate_up", "shared_gate", "shared_up", "sorted_rows")}
    values.update(_plan(problem["tall"], cap), tokens=TOKENS, rows=problem["total"], experts=EXPERTS,
                  act=torch.zeros(problem["total"], 512, dtype=torch.bfloat16, device="cuda"),
                  shared_act=torch.zeros(TOKENS, 512, dtype=torch.bfloat16, device="cuda"))
    values.update(changed)
    return product_probe.operands(**values), values


def _run(launch, operands, *arguments) -> None:
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert launch(ctypes.byref(operands), *arguments, ctypes.c_void_p(status.data_ptr()), LIMIT) == 0
    torch.cuda.synchronize()
    assert status.item() == 0


@pytest.mark.parametrize("with_shared", [0, 1])
@pytest.mark.parametrize("fetch", [0, 1], ids=["gathered", "fetched"])
def test_fed_rows_give_the_bits_of_the_one_sm_kernel(product_probe, feed_probe, problem, fetch, with_shared):
    want_operands, want = _operands(product_probe, problem, 128)
    _run(product_probe.run_gate_up, want_operands, 0, with_shared, problem["sms"])
    operands, got = _operands(product_probe, problem, 256)
    _run(feed_probe.run_gate_up_fed, operands, fetch, with_shared, problem["sms"])
    assert want["act"].float().abs().amax() > 0
    assert torch.equal(got["act"], want["act"])
    assert torch.equal(got["shared_act"], want["shared_act"])
    assert bool(want["shared_act"].any()) == bool(with_shared)


@pytest.mark.parametrize("with_shared", [0, 1])
@pytest.mark.parametrize("limit_ns", [0, 4_000, 12_000, 5_000_000])
def test_fetched_product_stops_and_recovers(product_probe, feed_probe, problem, limit_ns, with_shared):
    operands, held = _operands(product_probe, problem, 256)
    _check(lambda status, limit: feed_probe.run_gate_up_fed(ctypes.byref(operands), 1, with_shared, problem["sms"],
                                                            ctypes.c_void_p(status.data_ptr()), limit),
           held["act"], limit_ns, must_run_out=limit_ns == 0)


def test_fetched_rows_are_there_when_they_are_read(product_probe, feed_probe, problem):
    """The rows of a pair's second block are written by its own threads and read by products that the first block issues: 200
    launches in a row on two inputs in turn, so that a stage read too early would hold rows of another launch, K step or tile."""
    rounds, inputs = 200, [problem["x"], _normal(SEED + 9, TOKENS, 2048)]
    sides, held = [], []
    for x in inputs:
        operands, values = _operands(product_probe, problem, 256, x=x)
        _run(feed_probe.run_gate_up_fed, operands, 0, 1, problem["sms"])            # by TMA gathers
        sides.append(_operands(product_probe, problem, 256, x=x))
        held.append(values)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for index in range(rounds):
        operands, values = sides[index & 1]
        assert feed_probe.run_gate_up_fed(ctypes.byref(operands), 1, 1, problem["sms"], ctypes.c_void_p(status.data_ptr()), LIMIT) == 0
        torch.cuda.synchronize()
        wrong += (values["act"].view(torch.int16) != held[index & 1]["act"].view(torch.int16)).sum()
        wrong += (values["shared_act"].view(torch.int16) != held[index & 1]["shared_act"].view(torch.int16)).sum()
        values["act"].zero_()
        values["shared_act"].zero_()
        torch.cuda.synchronize()
    assert status.item() == 0
    assert int(wrong) == 0
    assert not torch.equal(held[0]["act"], held[1]["act"])


@pytest.mark.parametrize("tokens", [127, 128, 129, 130, 333, 4500])
def test_calls_on_either_side_of_the_limit_give_the_bits_of_the_copy(package, gpu_layers, synth, tokens):
    device = torch.device("cuda", 0)
    generator = torch.Generator().manual_seed(SEED + tokens)
    ids = torch.stack([torch.randperm(256, generator=generator)[:8] for _ in range(tokens)]).to(torch.int32)
    ids[:, 0] = 5                                                    # one expert with a row of every token
    routing = torch.rand(tokens, 8, generator=generator).to(torch.bfloat16).to(device)
    h2 = synth.activations(SEED, tokens, "input", 0).to(device)
    resid = synth.activations(SEED, tokens, "residual", 0).to(device)
    results = []
    for flags in (0, package.provider.FLAG_MATERIALIZED_DISPATCH):
        provider = package.MoeProvider(layers=1, max_prefill_tokens=tokens, flags=flags)
        try:
            provider.bind_layer(0, gpu_layers(0)["cuda"])
            provider.set_forced_routing(ids.to(device), routing)
            views, dbg = provider.make_debug(tokens, prefill=True, with_logits=False, with_slot_rows=True)
            out = provider.launch_selected_moe(post_attention=h2, residual_hidden=resid, model_layer=0, debug=views)
            provider.sync_metrics()
            results.append((out, dbg["slot_rows"], dbg["shared_scaled"]))
        finally:
            provider.release()
    for fed, copied in zip(*results):
        assert torch.equal(fed, copied)
