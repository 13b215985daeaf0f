"""GPU parity of the pair GEMM's tail tiles: the token rows past whole 256, as the n operand of tiles whose rows are features. Bounds as
elsewhere: helpers.rel_error <= 2e-2 (BF16 output) against the fp64 oracle fed the same quantised activations."""
import numpy as np
import pytest

import oracle
from augur_v100_b200 import abi, host, synth
from helpers import TOLERANCE, bits_from_torch_bf16, rel_error, torch_bf16_from_bits
from test_gpu_prefill import ctx  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


# One to 128 tokens in the tail (n of 32, 64, 96, 128; one and two chunks of either half), a half tile at the end of the weights (odd number of
# 128-row blocks), a partial last k block, tiles cut along k and not (a plan without scratch for it), several whole rounds ahead.
@pytest.mark.parametrize("cut", [True, False])
@pytest.mark.parametrize("rows,cols,tokens,terms", [(17408, 576, 257, 3), (17280, 832, 512 + 33, 2), (9600, 1088, 768 + 64, 3), (18944, 576, 256 + 65, 1),
                                                    (5120, 4352, 768 + 9, 3), (19072, 320, 1280 + 128, 3), (12416, 2624, 512 + 97, 1)])
def test_tail_tiles(ctx, rows, cols, tokens, terms, cut):  # noqa: F811
    plan = host.Plan(ctx["stream"], host.gemm_plan_scratch_bytes() if cut else 1 << 18)
    w_codes, w_scales, g_w = synth.make_weight(rows, 75, "w", rows, cols)
    x_bits = synth.make_activation(rows, 75, "x", tokens, cols)
    weight = host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(ctx["stream"], abi.LAYOUT_TCGEN05, rows, cols, w_codes, w_scales, g_w)
    linear = host.Nvfp4Sm100PrefillLinear.bind(plan, weight, torch_bf16_from_bits(x_bits, ctx["device"]), terms=terms)
    results = []
    for _ in range(6):      # the later launches find the plan's flags as the first left them
        linear.out.fill_(float("nan"))
        linear.submit_for_plan()
        ctx["stream"].synchronize()
        results.append(bits_from_torch_bf16(linear.out))
    assert plan.device_status() == 0
    assert all(np.array_equal(results[0], again) for again in results[1:])
    codes, scales = linear.staged_planes()
    whole = tokens // 256 * 256
    picked = sorted({0, whole - 1, whole, whole + 31, whole + 32, whole + 63, whole + 64, tokens - 2, tokens - 1} & set(range(tokens)))
    a64 = oracle.act_dequant_f64(np.ascontiguousarray(codes[:, picked]), np.ascontiguousarray(scales[:, picked]), 2.0 ** -8, len(picked), cols, terms)
    y64 = oracle.linear_f64_xf64(w_codes, w_scales, g_w, rows, cols, a64, threads=oracle.max_threads())
    assert rel_error(results[0].reshape(tokens, rows)[picked], y64) <= TOLERANCE
    plan.close()


# SwiGLU and the fused intermediate quantiser behind tail tiles: the block equals the one that quantises in a launch of its own, with and without
# the BF16 intermediate.
@pytest.mark.parametrize("hidden,inter,tokens,terms", [(512, 9600, 256 + 20, 3), (384, 9728, 512 + 128, 2), (640, 8704, 768 + 70, 1)])
def test_tail_tiles_quantise(ctx, hidden, inter, tokens, terms):  # noqa: F811
    torch = ctx["torch"]
    generator = torch.Generator(device=ctx["device"])
    generator.manual_seed(hidden + tokens)

    def planes(rows, cols):
        raw = torch.randn((rows, cols // 16), device=ctx["device"], generator=generator).abs() * 0.5
        return (torch.randint(0, 256, (rows, cols // 2), dtype=torch.uint8, device=ctx["device"], generator=generator),
                raw.clamp(2.0 ** -9, 448.0).to(torch.float8_e4m3fn).view(torch.uint8).clamp(1, 0x7E))

    torch.cuda.synchronize()
    plan = host.Plan(ctx["stream"], host.gemm_plan_scratch_bytes())
    repack = host.Nvfp4Sm100Weight.repack_device_planes
    gate_up = repack(ctx["stream"], abi.LAYOUT_TCGEN05, 2 * inter, hidden, *planes(2 * inter, hidden), synth.GLOBAL_SCALE)
    gate_up.global_scale_b = 1.5 * synth.GLOBAL_SCALE
    down = repack(ctx["stream"], abi.LAYOUT_TCGEN05, hidden, inter, *planes(hidden, inter), synth.GLOBAL_SCALE)
    x = torch.randn((tokens, hidden), device=ctx["device"], generator=generator).to(torch.bfloat16)
    torch.cuda.synchronize()
    programs = [host.Nvfp4Sm100PrefillFfnProgram.bind(plan, gate_up, down, x, terms=terms, intermediate_global_scale=2.0 ** -8, **options)
                for options in ({"fuse_quantiser": False}, {}, {"keep_intermediate": True})]
    for program in programs:
        program.out.fill_(float("nan"))
        program.intermediate.fill_(float("nan"))
        program.submit_for_plan()
    ctx["stream"].synchronize()
    assert plan.device_status() == 0
    assert bool(torch.isfinite(programs[0].out.float()).all()) and bool(torch.isfinite(programs[0].intermediate.float()).all())
    for program in programs[1:]:
        assert torch.equal(programs[0].out.view(torch.int16), program.out.view(torch.int16))
    assert torch.equal(programs[0].intermediate.view(torch.int16), programs[2].intermediate.view(torch.int16))
    plan.close()
