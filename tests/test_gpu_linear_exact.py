"""`Nvfp4Sm100Linear` on small batches of weights below the line of the large ones: every activation is multiplied as it is, however far below its
neighbours, and non-finite elements reach each output by the rules of IEEE arithmetic. Bound as elsewhere: helpers.rel_error <= 2e-2
against the fp64 oracle."""
import numpy as np
import pytest

import oracle
from augur_v100_b200 import host, synth
from helpers import TOLERANCE, bits_from_torch_bf16, rel_error, torch_bf16_from_bits
from test_gpu_small_token_tc import ctx  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu

SHAPES = [(1024, 5120, 1), (2048, 2048, 4), (1024, 4096, 8), (3968, 8704, 5)]


def _run(ctx, rows, cols, codes, scales, glob, x_bits):  # noqa: F811
    linear = host.Nvfp4Sm100Linear(ctx["stream"], rows, cols, codes, scales, glob)
    plan = host.Plan(ctx["stream"], max(host.gemv_scratch_bytes(rows, cols), host.gemv_tc_linear_scratch_bytes(cols)))
    binding = linear.bind(plan, torch_bf16_from_bits(x_bits, ctx["device"]))
    binding.submit_for_plan()
    ctx["stream"].synchronize()
    assert plan.device_status() == 0
    got = bits_from_torch_bf16(binding.out).reshape(x_bits.shape[0], rows)
    plan.close()
    return type(binding), got


# One element in every group of sixteen is 2^30 times the others and meets zero weights: the outputs are those of the small elements alone.
@pytest.mark.parametrize("rows,cols,tokens", SHAPES)
def test_wide_range_rows(ctx, rows, cols, tokens):  # noqa: F811
    codes, scales, glob = synth.make_weight(rows + tokens, 92, "w", rows, cols)
    codes[:, 3::8] &= 0xF0            # column 6 of every group
    x = np.random.default_rng(cols).standard_normal((tokens, cols)).astype(np.float32)
    x[:, 6::16] *= 2.0 ** 30
    x_bits = synth.f32_to_bf16_bits(x)
    kind, got = _run(ctx, rows, cols, codes, scales, glob, x_bits)
    y64 = oracle.linear_f64(codes, scales, glob, rows, cols, x_bits, threads=oracle.max_threads()).reshape(tokens, rows)
    assert rel_error(got, y64) <= TOLERANCE
    assert kind is host.Nvfp4Sm100Projection


# An infinity gives infinities of the weights' signs (NaN where it meets a zero weight), a NaN all NaN; the other rows are as ever.
@pytest.mark.parametrize("rows,cols,tokens", [(1024, 5120, 4), (1024, 4096, 8), (3968, 8704, 5)])
def test_non_finite_elements(ctx, rows, cols, tokens):  # noqa: F811
    codes, scales, glob = synth.make_weight(rows - tokens, 92, "w", rows, cols)
    column = cols - 40                # even: the low nibble
    x_bits = synth.make_activation(rows, 92, "x", tokens, cols)
    x_bits[1, column], x_bits[2, column], x_bits[3, 17] = 0x7F80, 0xFF80, 0x7FC0
    kind, got = _run(ctx, rows, cols, codes, scales, glob, x_bits)
    nibble = codes[:, column // 2] & 15
    zero, negative = (nibble & 7) == 0, nibble >= 8
    for row, flip in ((1, 0), (2, 1)):
        assert np.all((got[row][zero] & 0x7FFF) > 0x7F80)
        assert np.array_equal(got[row][~zero], np.where(negative[~zero] ^ bool(flip), 0xFF80, 0x7F80))
    assert np.all((got[3] & 0x7FFF) > 0x7F80)
    finite = [row for row in range(tokens) if row not in (1, 2, 3)]
    y64 = oracle.linear_f64(codes, scales, glob, rows, cols, np.ascontiguousarray(x_bits[finite]), threads=oracle.max_threads()).reshape(len(finite), rows)
    assert rel_error(got[finite], y64) <= TOLERANCE
    assert kind is host.Nvfp4Sm100Projection
