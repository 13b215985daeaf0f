"""GPU parity of the small-token linear on tensor memory, as one launch that forms its own digits and as two where a CTA has many chunks of many
token rows: one k step, ragged last k block and row slice, every cluster size, more tiles than places on the GPU, rows whose groups are far
apart in magnitude, non-finite rows, and projections of different shapes in turn on one plan. Bound as elsewhere: helpers.rel_error <= 2e-2
against the fp64 oracle."""
import numpy as np
import pytest

import oracle
from augur_v100_b200 import abi, host, synth
from helpers import TOLERANCE, bits_from_torch_bf16, rel_error, torch_bf16_from_bits
from test_gpu_small_token_tc import ctx  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


def _bind(ctx, rows, cols, tokens, seed, plan=None):  # noqa: F811
    codes, scales, glob = synth.make_weight(seed, 92, "w", rows, cols)
    x = np.random.default_rng(seed).standard_normal((tokens, cols)).astype(np.float32)
    x[:, : cols // 4] *= 2.0 ** -19       # groups that keep the smallest block scale and lose low digits, beside full ones
    x_bits = synth.f32_to_bf16_bits(x)
    weight = host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(ctx["stream"], abi.LAYOUT_TCGEN05, rows, cols, codes, scales, glob)
    projection = host.Nvfp4Sm100TcProjection.bind(plan or ctx["plan"], weight, torch_bf16_from_bits(x_bits, ctx["device"]))
    return projection, oracle.linear_f64(codes, scales, glob, rows, cols, x_bits, threads=oracle.max_threads())


# (128, 64): one MMA; 17408 columns: clusters of 8; 37 and 45 tiles: of 7 and 6; 49920 rows: 390 tiles, more than fit at once
@pytest.mark.parametrize("rows,cols,tokens", [(128, 64, 1), (128, 17408, 3), (4736, 2112, 8), (5760, 1600, 7), (9088, 1344, 5), (49920, 64, 2), (384, 320, 4)])
def test_split_linear_edges(ctx, rows, cols, tokens):  # noqa: F811
    projection, y64 = _bind(ctx, rows, cols, tokens, rows + cols)
    other, other64 = _bind(ctx, 256, 1024, 8, 5)
    results = []
    for _ in range(3):      # the other shape's split overwrites this one's in the plan's scratch in between
        projection.submit_for_plan()
        other.submit_for_plan()
        ctx["stream"].synchronize()
        results.append(bits_from_torch_bf16(projection.out))
    assert ctx["plan"].device_status() == 0
    assert rel_error(results[0], y64) <= TOLERANCE and all(np.array_equal(results[0], again) for again in results[1:])
    assert rel_error(bits_from_torch_bf16(other.out), other64) <= TOLERANCE


def _launches(projection):
    before = host.launch_count()
    projection.submit_for_plan()
    return host.launch_count() - before


# More than ten chunks of 256 columns per CTA and six token rows or more: a launch of its own forms the digits. 20800 columns: clusters of 8 with 11
# chunks, the last of one k step; 5120 x 17408: clusters of 6; 34816 rows: whole tiles of 12. Ten chunks (20480 columns) or five token rows: one launch.
@pytest.mark.parametrize("rows,cols,tokens,launches", [(128, 20800, 8, 2), (256, 24640, 6, 2), (5120, 17408, 7, 2), (34816, 2880, 8, 2),
                                                       (128, 20480, 8, 1), (128, 20800, 5, 1)])
def test_digits_of_a_launch_ahead(ctx, rows, cols, tokens, launches):  # noqa: F811
    plan = host.Plan(ctx["stream"], host.gemv_tc_linear_scratch_bytes(max(cols, 20736)))      # not a byte more
    projection, y64 = _bind(ctx, rows, cols, tokens, rows + cols, plan)
    other, other64 = _bind(ctx, 128, 20736, 6, 11, plan)
    results = []
    for _ in range(3):      # the other shape's digits overwrite this one's in the plan's scratch in between
        projection.out.fill_(float("nan"))
        assert _launches(projection) == launches and _launches(other) == 2
        ctx["stream"].synchronize()
        results.append(bits_from_torch_bf16(projection.out))
    assert plan.device_status() == 0
    assert rel_error(results[0], y64) <= TOLERANCE and all(np.array_equal(results[0], again) for again in results[1:])
    assert rel_error(bits_from_torch_bf16(other.out), other64) <= TOLERANCE
    plan.close()


# The largest BF16 exponents (one element of a row far above the rest) and the smallest, subnormal rows among them, with block
# and global scales that keep the sums inside F32 and the outputs normal.
@pytest.mark.parametrize("rows,cols,launches", [(256, 1088, 1), (128, 20800, 2)])
@pytest.mark.parametrize("exponents,block_scale,glob", [((122, 123, 124, 125, 126, 127), 0x18, 1.0 / 448.0),
                                                        ((-86, -88, -99, -110, -124, -130), 0x70, 24.0)])
def test_split_covers_every_exponent(ctx, exponents, block_scale, glob, rows, cols, launches):  # noqa: F811
    generator = np.random.default_rng(block_scale)
    codes = generator.integers(0, 256, (rows, cols // 2), dtype=np.uint8)
    scales = np.full((rows, cols // 16), block_scale, dtype=np.uint8)
    x = generator.standard_normal((len(exponents), cols)) * 2.0 ** (np.array(exponents)[:, None] - 8)
    x[:, 700] = 1.5 * 2.0 ** np.array(exponents)
    x_bits = synth.f32_to_bf16_bits(x.astype(np.float32))
    weight = host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(ctx["stream"], abi.LAYOUT_TCGEN05, rows, cols, codes, scales, glob)
    plan = host.Plan(ctx["stream"], host.gemv_tc_linear_scratch_bytes(cols))
    projection = host.Nvfp4Sm100TcProjection.bind(plan, weight, torch_bf16_from_bits(x_bits, ctx["device"]))
    assert _launches(projection) == launches
    ctx["stream"].synchronize()
    assert plan.device_status() == 0
    y64 = oracle.linear_f64(codes, scales, glob, rows, cols, x_bits, threads=oracle.max_threads()).reshape(len(exponents), rows)
    got = bits_from_torch_bf16(projection.out).reshape(len(exponents), rows)
    for row, exponent in enumerate(exponents):
        assert rel_error(got[row], y64[row]) <= TOLERANCE, exponent
    plan.close()


# An infinity or a NaN makes its row NaN, whichever part of k holds it, and no other row.
@pytest.mark.parametrize("rows,cols,tokens,launches", [(384, 4160, 6, 1), (128, 20800, 6, 2)])
def test_non_finite_rows(ctx, rows, cols, tokens, launches):  # noqa: F811
    codes, scales, glob = synth.make_weight(21, 92, "w", rows, cols)
    x = np.random.default_rng(21).standard_normal((tokens, cols)).astype(np.float32)
    x[1, 0], x[3, cols - 1], x[4, 2000] = np.inf, -np.inf, np.nan
    x_bits = synth.f32_to_bf16_bits(x)
    x_bits[4, 2000] = 0x7FC0       # rounding a NaN is not what is tested
    weight = host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(ctx["stream"], abi.LAYOUT_TCGEN05, rows, cols, codes, scales, glob)
    plan = host.Plan(ctx["stream"], host.gemv_tc_linear_scratch_bytes(cols))
    projection = host.Nvfp4Sm100TcProjection.bind(plan, weight, torch_bf16_from_bits(x_bits, ctx["device"]))
    assert _launches(projection) == launches
    ctx["stream"].synchronize()
    assert plan.device_status() == 0
    got = bits_from_torch_bf16(projection.out).reshape(tokens, rows)
    assert np.all((got[[1, 3, 4]] & 0x7FFF) > 0x7F80)
    finite = [0, 2, 5]
    y64 = oracle.linear_f64(codes, scales, glob, rows, cols, np.ascontiguousarray(x_bits[finite]), threads=oracle.max_threads())
    assert rel_error(got[finite], y64.reshape(3, rows)) <= TOLERANCE
    plan.close()


# `Nvfp4Sm100Linear` binds this kernel for large weights.
def test_linear_dispatch_by_size(ctx):  # noqa: F811
    rows, cols, tokens = 32768, 1024, 6
    codes, scales, glob = synth.make_weight(7, 95, "w", rows, cols)
    x_bits = synth.make_activation(7, 95, "x", tokens, cols)
    linear = host.Nvfp4Sm100Linear(ctx["stream"], rows, cols, codes, scales, glob)
    plan = host.Plan(ctx["stream"], 1 << 20)
    binding = linear.bind(plan, torch_bf16_from_bits(x_bits, ctx["device"]))
    binding.submit_for_plan()
    ctx["stream"].synchronize()
    y64 = oracle.linear_f64(codes, scales, glob, rows, cols, x_bits, threads=oracle.max_threads())
    assert plan.device_status() == 0 and isinstance(binding, host.Nvfp4Sm100TcProjection)
    assert rel_error(bits_from_torch_bf16(binding.out), y64) <= TOLERANCE
    plan.close()


# A plan of one byte less than the kernel's scratch keeps the general kernel, as does a weight of more rows than the kernel takes; a
# fault of the binding itself is raised and does not change the kernel.
def test_linear_dispatch_by_scratch_rows_and_faults(ctx):  # noqa: F811
    rows, cols, tokens = 32768, 1024, 5
    codes, scales, glob = synth.make_weight(8, 95, "w", rows, cols)
    linear = host.Nvfp4Sm100Linear(ctx["stream"], rows, cols, codes, scales, glob)
    x_bits = synth.make_activation(8, 95, "x", tokens, cols)
    x = torch_bf16_from_bits(x_bits, ctx["device"])
    y64 = oracle.linear_f64(codes, scales, glob, rows, cols, x_bits, threads=oracle.max_threads())
    need = host.gemv_tc_linear_scratch_bytes(cols)
    small_need = host.gemv_scratch_bytes(rows, cols)
    enough = host.Plan(ctx["stream"], need)
    binding = linear.bind(enough, x)
    assert isinstance(binding, host.Nvfp4Sm100TcProjection)
    binding.submit_for_plan()
    ctx["stream"].synchronize()
    assert rel_error(bits_from_torch_bf16(binding.out), y64) <= TOLERANCE
    less = host.Plan(ctx["stream"], need - 256)
    with pytest.raises(host.CudaRuntimeError):
        host.Nvfp4Sm100TcProjection.bind(less, linear.wide, x)
    assert not linear._on_tensor_memory(less, tokens)
    roomy = host.Plan(ctx["stream"], max(need, small_need))
    linear.wide.global_scale = float("nan")       # concerns this kernel's copy of the weight only
    with pytest.raises(host.CudaRuntimeError):
        linear.bind(roomy, x)
    for plan in (enough, less, roomy):
        plan.close()
    rows, cols = (1 << 18) + 128, 128
    codes, scales, glob = synth.make_weight(9, 95, "w", rows, cols)
    linear = host.Nvfp4Sm100Linear(ctx["stream"], rows, cols, codes, scales, glob)
    x_bits = synth.make_activation(9, 95, "x", tokens, cols)
    plan = host.Plan(ctx["stream"], host.gemv_scratch_bytes(rows, cols))
    binding = linear.bind(plan, torch_bf16_from_bits(x_bits, ctx["device"]))
    binding.submit_for_plan()
    ctx["stream"].synchronize()
    y64 = oracle.linear_f64(codes, scales, glob, rows, cols, x_bits, threads=oracle.max_threads())
    assert type(binding) is host.Nvfp4Sm100Projection and rel_error(bits_from_torch_bf16(binding.out), y64) <= TOLERANCE
    plan.close()
