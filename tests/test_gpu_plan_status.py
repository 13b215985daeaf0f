"""What a launch that gave up leaves in a plan is gone once the plan's status has been read. The failure is planted from the host, in the plan's
memory: a status word and counters and flags as such a launch may leave them."""
import numpy as np
import pytest

from augur_v100_b200 import abi, host, synth
from helpers import bits_from_torch_bf16, torch_bf16_from_bits
from test_gpu_prefill import ctx  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu

COUNTER_WORDS = 2 * 16384


def _words(torch, address, count):
    holder = type("Words", (), {"__cuda_array_interface__": {"shape": (count,), "typestr": "<i4", "data": (address, False), "version": 3}})()
    return torch.as_tensor(holder, device="cuda")


def test_status_read_clears_flags(ctx):  # noqa: F811
    torch = ctx["torch"]
    rows, cols, tokens = 2816, 5248, 793       # tiles cut along k, their parts handed over by flags
    plan = host.Plan(ctx["stream"], host.gemm_plan_scratch_bytes())
    scratch = plan.snapshot().scratch
    codes, scales, glob = synth.make_weight(3, 75, "w", rows, cols)
    weight = host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(ctx["stream"], abi.LAYOUT_TCGEN05, rows, cols, codes, scales, glob)
    x_bits = synth.make_activation(3, 75, "x", tokens, cols)
    linear = host.Nvfp4Sm100PrefillLinear.bind(plan, weight, torch_bf16_from_bits(x_bits, ctx["device"]), terms=3)
    linear.submit_for_plan()
    ctx["stream"].synchronize()
    wanted = bits_from_torch_bf16(linear.out)
    counters, status = _words(torch, scratch, COUNTER_WORDS), _words(torch, scratch - 256, 1)
    assert plan.device_status() == 0 and int(counters.abs().sum()) == 0
    counters[::5] = 1
    counters[-1] = 7
    status.fill_(0x107)
    torch.cuda.synchronize()
    assert plan.device_status() == 0x107
    assert int(counters.abs().sum()) == 0
    linear.submit_for_plan()
    ctx["stream"].synchronize()
    assert np.array_equal(bits_from_torch_bf16(linear.out), wanted) and int(counters.abs().sum()) == 0
    plan.close()


def test_status_read_stays_inside_a_small_plan(ctx):  # noqa: F811
    torch = ctx["torch"]
    plan = host.Plan(ctx["stream"], 512)
    scratch = plan.snapshot().scratch
    words, status = _words(torch, scratch, 128), _words(torch, scratch - 256, 1)
    words.fill_(3)
    status.fill_(0x107)
    torch.cuda.synchronize()
    assert plan.device_status() == 0x107 and int(words.abs().sum()) == 0
    plan.close()
