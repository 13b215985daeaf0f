"""GPU parity of the prefill GEMM's two kernels over token counts: the narrow kernel, token pairs alone, and
pairs with tail tiles; half tiles of an odd number of 128-row weight blocks. Bounds as elsewhere:
helpers.rel_error <= 2e-2 (BF16 output) against the fp64 oracle fed the same quantised activations."""
import numpy as np
import pytest

import oracle
from augur_v100_b200 import abi, host, synth
from helpers import TOLERANCE, bits_from_torch_bf16, rel_error, torch_bf16_from_bits
from test_gpu_prefill import _check_gemm, ctx  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def split_plan(ctx):  # noqa: F811
    plan = host.Plan(ctx["stream"], host.gemm_plan_scratch_bytes())   # room to cut leftover tiles
    yield plan
    plan.close()


# One MMA; partial last k block; MMA n of 16, 32, 128; two token tiles, the second of one token; several CTAs per tile up to the
# largest cluster; more tiles than CTAs at once (390 items).
@pytest.mark.parametrize("rows,cols,tokens,terms", [(128, 64, 9, 1), (384, 192, 16, 3), (128, 320, 17, 2), (2944, 2112, 127, 3),
                                                    (256, 832, 128, 1), (640, 1088, 129, 3), (128, 17408, 33, 2), (49920, 64, 40, 2)])
def test_narrow_token_ranges(ctx, rows, cols, tokens, terms):  # noqa: F811
    assert _check_gemm(ctx, rows, cols, tokens, terms, seed=rows + tokens) <= TOLERANCE


# The same on weights that stay with the narrow kernel by a margin (tests/test_pair_work_cpu.py asks the library's rule for these and those above): more tiles than
# places, 301 and 390 of them, MMA n of 16, 48, 112 and 128, two and five token tiles, clusters of up to eight.
NARROW = [(38528, 832, 9, 1), (49920, 1088, 16, 1), (49920, 2112, 40, 2), (384, 4352, 112, 2), (1152, 5120, 128, 1), (640, 4352, 200, 1), (512, 4352, 577, 1)]


@pytest.mark.parametrize("rows,cols,tokens,terms", NARROW)
def test_narrow_tiles(ctx, rows, cols, tokens, terms):  # noqa: F811
    assert _check_gemm(ctx, rows, cols, tokens, terms, seed=rows + tokens) <= TOLERANCE


# Token pairs with a half tile at the end (one round; several rounds; fewer tiles than pairs),
# pairs with tail tiles of 44 tokens.
@pytest.mark.parametrize("rows,cols,tokens,terms", [(17280, 576, 530, 3), (19072, 832, 1500, 1), (4992, 4352, 400, 3), (17408, 5120, 300, 3)])
def test_pair_tiles_and_tails(ctx, split_plan, rows, cols, tokens, terms):  # noqa: F811
    w_codes, w_scales, g_w = synth.make_weight(rows, 74, "w", rows, cols)
    x_bits = synth.make_activation(rows, 74, "x", tokens, cols)
    weight = host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(ctx["stream"], abi.LAYOUT_TCGEN05, rows, cols, w_codes, w_scales, g_w)
    linear = host.Nvfp4Sm100PrefillLinear.bind(split_plan, weight, torch_bf16_from_bits(x_bits, ctx["device"]), terms=terms)
    results = []
    for _ in range(3):      # the later launches find the plan's flags as the first left them
        linear.out.fill_(float("nan"))
        linear.submit_for_plan()
        ctx["stream"].synchronize()
        results.append(bits_from_torch_bf16(linear.out))
    assert split_plan.device_status() == 0
    assert all(np.array_equal(results[0], again) for again in results[1:])
    codes, scales = linear.staged_planes()
    picked = sorted({0, 127, 128, 255, 256, 257, tokens // 2, tokens - 2, tokens - 1})     # edges of the tiles
    a64 = oracle.act_dequant_f64(np.ascontiguousarray(codes[:, picked]), np.ascontiguousarray(scales[:, picked]), 2.0 ** -8, len(picked), cols, terms)
    y64 = oracle.linear_f64_xf64(w_codes, w_scales, g_w, rows, cols, a64, threads=oracle.max_threads())
    assert rel_error(results[0].reshape(tokens, rows)[picked], y64) <= TOLERANCE


# The fused intermediate quantiser in both kernels' epilogues: the whole block equals the one that quantises in a launch of its own.
@pytest.mark.parametrize("hidden,inter,tokens", [(256, 640, 20), (384, 1152, 200), (5120, 8704, 300), (1536, 1408, 825)])
def test_fused_quantiser_in_every_kernel(ctx, split_plan, hidden, inter, tokens):  # noqa: F811
    torch = ctx["torch"]
    generator = torch.Generator(device=ctx["device"])
    generator.manual_seed(hidden + tokens)

    def planes(rows, cols):
        raw = torch.randn((rows, cols // 16), device=ctx["device"], generator=generator).abs() * 0.5
        return (torch.randint(0, 256, (rows, cols // 2), dtype=torch.uint8, device=ctx["device"], generator=generator),
                raw.clamp(2.0 ** -9, 448.0).to(torch.float8_e4m3fn).view(torch.uint8).clamp(1, 0x7E))

    torch.cuda.synchronize()
    repack = host.Nvfp4Sm100Weight.repack_device_planes
    gate_up = repack(ctx["stream"], abi.LAYOUT_TCGEN05, 2 * inter, hidden, *planes(2 * inter, hidden), synth.GLOBAL_SCALE)
    gate_up.global_scale_b = 1.5 * synth.GLOBAL_SCALE
    down = repack(ctx["stream"], abi.LAYOUT_TCGEN05, hidden, inter, *planes(hidden, inter), synth.GLOBAL_SCALE)
    x = torch.randn((tokens, hidden), device=ctx["device"], generator=generator).to(torch.bfloat16)
    torch.cuda.synchronize()
    programs = [host.Nvfp4Sm100PrefillFfnProgram.bind(split_plan, gate_up, down, x, terms=3, intermediate_global_scale=2.0 ** -8, fuse_quantiser=fuse)
                for fuse in (False, True)]
    for program in programs:
        program.out.fill_(float("nan"))
        program.submit_for_plan()
    ctx["stream"].synchronize()
    assert split_plan.device_status() == 0
    assert bool(torch.isfinite(programs[0].out.float()).all())
    assert torch.equal(programs[0].out.view(torch.int16), programs[1].out.view(torch.int16))
