"""GPU parity of the pair GEMM's tail tiles, the token rows past whole 256 as the n operand of tiles whose rows are features, and of leftover tiles cut
along k. Bounds as elsewhere: helpers.rel_error <= 2e-2 (BF16 output) against the fp64 oracle fed the same quantised activations."""
import numpy as np
import pytest

import oracle
from augur_v100_b200 import abi, host, synth
from helpers import TOLERANCE, bits_from_torch_bf16, rel_error, torch_bf16_from_bits
from test_gpu_prefill import ctx  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


# rows, cols, tokens, terms; tail columns of a launch whose plan has room to cut tiles and whether tail tiles are cut then; tail columns without the room
# (0: another path). tests/test_pair_work_cpu.py asks the library's rule for them.
# One to 128 tokens in the tail (n of 32, 64, 96, 128; one and two chunks of either half), a half tile at the end of the weights (odd number of
# 128-row blocks), a partial last k block, several whole rounds ahead, parts handed over of either chunk.
CASES = [(17408, 576, 257, 3, 32, False, 32), (17280, 832, 512 + 33, 2, 64, False, 64), (9600, 1088, 768 + 64, 3, 64, False, 64),
         (18944, 576, 256 + 65, 1, 0, False, 0), (5120, 4352, 768 + 9, 3, 0, False, 0), (19072, 320, 1280 + 128, 3, 0, False, 0), (12416, 2624, 512 + 97, 1, 0, False, 0),
         (18560, 2240, 256 + 57, 1, 64, False, 64), (6016, 1280, 768 + 65, 3, 96, False, 96), (8832, 1856, 512 + 121, 3, 128, False, 128),
         (2816, 5248, 768 + 25, 3, 32, True, 0), (8320, 2112, 1024 + 44, 3, 64, True, 64), (6144, 2624, 1024 + 44, 3, 64, True, 0),
         (7808, 3456, 1024 + 57, 2, 64, True, 64), (6272, 3264, 1024 + 65, 3, 96, True, 0), (7808, 5056, 1024 + 96, 1, 96, True, 0),
         (7680, 2176, 1024 + 121, 3, 128, True, 0), (6016, 4160, 1024 + 128, 2, 128, True, 0)]


@pytest.mark.parametrize("cut", [True, False])
@pytest.mark.parametrize("rows,cols,tokens,terms", [case[:4] for case in CASES])
def test_tail_tiles(ctx, rows, cols, tokens, terms, cut):  # noqa: F811
    _check(ctx, rows, cols, tokens, terms, cut)


# Leftover tiles without a tail: fewer tiles than pairs, one round and two; as many parts of every tile, and shares that are parts of two tiles (74 pairs).
# rows, cols, tokens, terms; pairs that share them (0: the narrow kernel's).
LEFTOVER = [(768, 12032, 1895, 1, 72), (768, 9728, 1895, 1, 0), (768, 5248, 1974, 2, 72), (1024, 7744, 2363, 2, 74), (768, 4864, 1942, 3, 72), (1280, 6528, 1921, 3, 74),
            (2176, 6720, 2286, 1, 14), (3200, 8640, 2198, 1, 74), (2176, 4096, 2370, 2, 32), (3712, 4864, 1961, 2, 74), (2688, 2368, 2205, 3, 50),
            (3200, 2880, 2127, 3, 74), (4480, 7104, 2366, 1, 64), (4224, 3968, 2399, 2, 44), (4224, 2240, 2372, 3, 44), (5376, 3584, 2190, 3, 74)]


@pytest.mark.parametrize("rows,cols,tokens,terms", [case[:4] for case in LEFTOVER])
def test_leftover_tiles(ctx, rows, cols, tokens, terms):  # noqa: F811
    _check(ctx, rows, cols, tokens, terms, True)


def _check(ctx, rows, cols, tokens, terms, cut):  # noqa: F811
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
    picked = sorted({0, tokens // 3, tokens // 2, whole - 129, whole - 1, whole, whole + 31, whole + 32, whole + 63, whole + 64, tokens - 2, tokens - 1} & set(range(tokens)))
    a64 = oracle.act_dequant_f64(np.ascontiguousarray(codes[:, picked]), np.ascontiguousarray(scales[:, picked]), 2.0 ** -8, len(picked), cols, terms)
    y64 = oracle.linear_f64_xf64(w_codes, w_scales, g_w, rows, cols, a64, threads=oracle.max_threads())
    assert rel_error(results[0].reshape(tokens, rows)[picked], y64) <= TOLERANCE
    plan.close()


# SwiGLU and the fused intermediate quantiser behind tail tiles, whole and cut along k: the block equals the one that quantises in a launch of its own, with
# and without the BF16 intermediate, and the latter is the oracle's of the same quantised input. hidden, inter, tokens, terms; of the gate|up GEMM: tail
# columns, cut or not.
BLOCKS = [(512, 9600, 256 + 20, 3, 0, False), (384, 9728, 512 + 128, 2, 0, False), (640, 8704, 768 + 70, 1, 0, False),
          (1920, 7040, 1024 + 32, 1, 32, False), (1152, 2176, 1024 + 44, 2, 64, False), (1152, 2944, 768 + 76, 3, 96, False), (2048, 4608, 1024 + 121, 3, 128, False),
          (896, 6656, 1024 + 31, 3, 32, True), (2816, 3840, 1024 + 63, 3, 64, True), (4096, 3968, 1024 + 63, 2, 64, True), (2944, 3968, 1024 + 89, 3, 96, True),
          (1024, 6784, 1024 + 128, 3, 128, True)]


# Leftover tiles of the gate|up GEMM cut along k, without a tail. hidden, inter, tokens, terms; pairs that share them.
LEFTOVER_BLOCKS = [(7424, 1280, 980, 3, 74), (7424, 1408, 2339, 1, 72), (3968, 1280, 2231, 2, 32), (7296, 1408, 2202, 2, 74), (2688, 1152, 2358, 3, 32),
                   (2816, 2816, 1887, 3, 56)]


@pytest.mark.parametrize("hidden,inter,tokens,terms", [case[:4] for case in BLOCKS + LEFTOVER_BLOCKS])
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
    both = planes(2 * inter, hidden)
    gate_up = repack(ctx["stream"], abi.LAYOUT_TCGEN05, 2 * inter, hidden, *both, synth.GLOBAL_SCALE)
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
    quantised = host.Nvfp4Sm100PrefillLinear.bind(plan, gate_up, x, terms=terms)
    quantised.submit_quant()
    ctx["stream"].synchronize()
    codes, scales = quantised.staged_planes()
    whole = tokens // 256 * 256
    picked = sorted({0, tokens // 3, tokens // 2, whole - 129, whole - 1, whole, whole + 31, whole + 32, whole + 63, whole + 64, whole + 95, whole + 96, tokens - 1} & set(range(tokens)))
    a64 = oracle.act_dequant_f64(np.ascontiguousarray(codes[:, picked]), np.ascontiguousarray(scales[:, picked]), 2.0 ** -8, len(picked), hidden, terms)
    sums = oracle.linear_f64_xf64(both[0].cpu().numpy(), both[1].cpu().numpy(), 1.0, 2 * inter, hidden, a64, threads=oracle.max_threads())
    sums = sums.reshape(len(picked), inter // 16, 2, 16)
    gate, up = sums[:, :, 0] * gate_up.global_scale, sums[:, :, 1] * gate_up.global_scale_b
    h64 = (gate / (1.0 + np.exp(-gate)) * up).reshape(len(picked), inter)
    assert rel_error(bits_from_torch_bf16(programs[2].intermediate[picked]), h64) <= TOLERANCE
    plan.close()
