"""GPU parity of the pair GEMM's tail tiles: the token rows past whole 256, as the n operand of tiles whose rows are features. Bounds as
elsewhere: helpers.rel_error <= 2e-2 (BF16 output) against the fp64 oracle fed the same quantised activations."""
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
         (18944, 576, 256 + 65, 1, 96, False, 96), (19072, 320, 1280 + 128, 3, 128, False, 128), (12416, 2624, 512 + 97, 1, 0, False, 0),
         (5120, 4352, 768 + 9, 3, 32, True, 0), (2048, 4160, 768 + 63, 3, 64, True, 0), (2432, 3776, 512 + 64, 3, 64, True, 0),
         (6400, 1856, 768 + 57, 2, 64, True, 0), (6272, 1856, 768 + 95, 3, 96, True, 0), (6272, 3904, 768 + 96, 1, 96, True, 0),
         (2688, 4992, 512 + 127, 3, 128, True, 0), (10496, 3264, 768 + 121, 1, 128, True, 128)]


@pytest.mark.parametrize("cut", [True, False])
@pytest.mark.parametrize("rows,cols,tokens,terms", [case[:4] for case in CASES])
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


# SwiGLU and the fused intermediate quantiser behind tail tiles, whole and cut along k: the block equals the one that quantises in a launch of its own, with
# and without the BF16 intermediate, and the latter is the oracle's of the same quantised input. hidden, inter, tokens, terms; of the gate|up GEMM: tail
# columns, cut or not.
BLOCKS = [(512, 9600, 256 + 20, 3, 32, False), (384, 9728, 512 + 128, 2, 128, False), (640, 8704, 768 + 70, 1, 96, False),
          (1920, 3328, 768 + 44, 2, 64, True), (4480, 896, 768 + 44, 3, 64, True), (3712, 896, 768 + 65, 3, 96, True), (4992, 1408, 768 + 121, 2, 128, True),
          (3456, 3200, 768 + 95, 1, 96, True)]


@pytest.mark.parametrize("hidden,inter,tokens,terms", [case[:4] for case in BLOCKS])
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
    picked = sorted({0, whole - 1, whole, whole + 31, whole + 32, whole + 63, whole + 64, whole + 95, whole + 96, tokens - 1} & set(range(tokens)))
    a64 = oracle.act_dequant_f64(np.ascontiguousarray(codes[:, picked]), np.ascontiguousarray(scales[:, picked]), 2.0 ** -8, len(picked), hidden, terms)
    sums = oracle.linear_f64_xf64(both[0].cpu().numpy(), both[1].cpu().numpy(), 1.0, 2 * inter, hidden, a64, threads=oracle.max_threads())
    sums = sums.reshape(len(picked), inter // 16, 2, 16)
    gate, up = sums[:, :, 0] * gate_up.global_scale, sums[:, :, 1] * gate_up.global_scale_b
    h64 = (gate / (1.0 + np.exp(-gate)) * up).reshape(len(picked), inter)
    assert rel_error(bits_from_torch_bf16(programs[2].intermediate[picked]), h64) <= TOLERANCE
    plan.close()
