"""GPU parity of the pair GEMM where its two rings (weight stages, token slots) wrap, against each other and from tile to tile:
k blocks below, at and above both depths, partial last k blocks, every number of activation terms, three tiles per CTA pair.
Bound as elsewhere: helpers.rel_error <= 2e-2 (BF16 output) against the fp64 oracle fed the same quantised activations."""
import numpy as np
import pytest

import oracle
from augur_v100_b200 import abi, host, synth
from helpers import TOLERANCE, bits_from_torch_bf16, rel_error, torch_bf16_from_bits
from test_gpu_prefill import ctx  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu
ROWS, TOKENS = 19072, 600


@pytest.mark.parametrize("cols,terms", [(448, 2), (512, 3), (768, 2), (832, 3), (1280, 1), (1344, 1), (2048, 2), (2112, 3)])
def test_rings_wrap(ctx, cols, terms):  # noqa: F811
    w_codes, w_scales, g_w = synth.make_weight(cols, 75, "w", ROWS, cols)
    x_bits = synth.make_activation(cols, 75, "x", TOKENS, cols)
    weight = host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(ctx["stream"], abi.LAYOUT_TCGEN05, ROWS, cols, w_codes, w_scales, g_w)
    plan = host.Plan(ctx["stream"], host.gemm_plan_scratch_bytes())
    linear = host.Nvfp4Sm100PrefillLinear.bind(plan, weight, torch_bf16_from_bits(x_bits, ctx["device"]), terms=terms)
    results = []
    for _ in range(2):
        linear.out.fill_(float("nan"))
        linear.submit_for_plan()
        ctx["stream"].synchronize()
        results.append(bits_from_torch_bf16(linear.out))
    assert plan.device_status() == 0
    assert np.array_equal(*results)
    codes, scales = linear.staged_planes()
    picked = [0, 127, 128, 255, 256, 511, 512, TOKENS - 1]
    a64 = oracle.act_dequant_f64(np.ascontiguousarray(codes[:, picked]), np.ascontiguousarray(scales[:, picked]), 2.0 ** -8, len(picked), cols, terms)
    y64 = oracle.linear_f64_xf64(w_codes, w_scales, g_w, ROWS, cols, a64, threads=oracle.max_threads())
    assert rel_error(results[0].reshape(TOKENS, ROWS)[picked], y64) <= TOLERANCE
