"""GPU parity of the mma.sync small-token kernel at the edges of its split: row groups dealt out to clusters of every size, ranges
of unequal length, slabs of unequal k, more warps than blocks, the split through scratch beside them, and every token count (the
staging differs by it). Bound as elsewhere: helpers.rel_error <= 2e-2 against the fp64 oracle; two submits give the same bits."""
import numpy as np
import pytest

import oracle
from augur_v100_b200 import abi, host, synth
from helpers import TOLERANCE, bits_from_torch_bf16, rel_error, torch_bf16_from_bits
from test_gpu_small_token import ctx  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


# 1 group; fewer blocks than warps; 33 and 75 groups over clusters with unequal slabs; 160 groups; 9 slabs, through scratch
@pytest.mark.parametrize("rows,cols,tokens", [(32, 128, 1), (32, 5120, 8), (64, 1152, 2), (1056, 5248, 3), (2400, 2176, 4), (5120, 5120, 5),
                                              (1024, 41600, 6), (17408, 256, 7)])
def test_cluster_split(ctx, rows, cols, tokens):  # noqa: F811
    codes, scales, glob = synth.make_weight(rows + cols, 93, "w", rows, cols)
    x_bits = synth.make_activation(rows + cols, 93, "x", tokens, cols)
    weight = host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(ctx["stream"], abi.LAYOUT_STREAM, rows, cols, codes, scales, glob)
    plan = host.Plan(ctx["stream"], host.gemv_scratch_bytes(rows, cols))
    projection = host.Nvfp4Sm100Projection.bind(plan, weight, torch_bf16_from_bits(x_bits, ctx["device"]))
    results = []
    for _ in range(2):
        projection.out.fill_(float("nan"))
        projection.submit_for_plan()
        ctx["stream"].synchronize()
        results.append(bits_from_torch_bf16(projection.out))
    assert plan.device_status() == 0
    plan.close()
    assert np.array_equal(*results)
    assert rel_error(results[0], oracle.linear_f64(codes, scales, glob, rows, cols, x_bits, threads=oracle.max_threads())) <= TOLERANCE


# many row groups per CTA, whose shares the warps add a group each: 10, 9 and 8 per CTA, a short last one, groups that straddle warps;
# 9 per cluster of four CTAs
@pytest.mark.parametrize("rows,cols,tokens", [(47360, 384, 8), (42560, 640, 3), (37888, 256, 1), (9504, 5120, 8)])
def test_many_groups_per_cta(ctx, rows, cols, tokens):  # noqa: F811
    test_cluster_split(ctx, rows, cols, tokens)


# members of a norm group whose ranges straddle clusters, one of them trimmed
@pytest.mark.parametrize("cols,rows,stored", [(1024, (1056, 64, 2080), (0, 48, 0)), (2560, (64, 64, 32, 96), (48, 48, 0, 0)), (5120, (4000,), (0,))])
def test_group_members_straddle_clusters(ctx, cols, rows, stored):  # noqa: F811
    torch, tokens = ctx["torch"], 6
    made = [synth.make_weight(cols + i, 94, "w", r, cols) for i, r in enumerate(rows)]
    weights = [host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(ctx["stream"], abi.LAYOUT_STREAM, r, cols, *planes) for r, planes in zip(rows, made)]
    plan = host.Plan(ctx["stream"], 64 << 20)
    x = torch.from_numpy(np.random.default_rng(cols).standard_normal((tokens, cols)).astype(np.float32)).to(ctx["device"])
    gain = torch.ones(cols, dtype=torch.float32, device=ctx["device"])
    torch.cuda.synchronize()
    program = host.Nvfp4Sm100NormGroupProgram.bind(plan, weights, x, gain, stored_rows=list(stored))
    program.submit_for_plan()
    ctx["stream"].synchronize()
    assert plan.device_status() == 0
    plan.close()
    staged = bits_from_torch_bf16(program.staged)
    for out, r, keep, planes in zip(program.outputs, rows, stored, made):
        y64 = oracle.linear_f64(*planes, r, cols, staged, threads=oracle.max_threads())
        assert rel_error(bits_from_torch_bf16(out), np.ascontiguousarray(y64.reshape(tokens, r)[:, : keep or r])) <= TOLERANCE


# Scratch that holds the members' slots when every member has its share of the SMs, but not the slots of all SMs over the union
# of the members' row groups: such a plan is enough. In clusters, which need no slots; nine slabs, through scratch.
@pytest.mark.parametrize("cols,rows,scratch", [(10496, (768, 768), 594176), (41728, (160, 160, 160), 1075200)])
def test_group_in_little_scratch(ctx, cols, rows, scratch):  # noqa: F811
    torch, tokens = ctx["torch"], 5
    made = [synth.make_weight(cols + i, 96, "w", r, cols) for i, r in enumerate(rows)]
    weights = [host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(ctx["stream"], abi.LAYOUT_STREAM, r, cols, *planes) for r, planes in zip(rows, made)]
    x = torch.from_numpy(np.random.default_rng(cols).standard_normal((tokens, cols)).astype(np.float32)).to(ctx["device"])
    gain = torch.ones(cols, dtype=torch.float32, device=ctx["device"])
    torch.cuda.synchronize()
    plan = host.Plan(ctx["stream"], scratch)
    program = host.Nvfp4Sm100NormGroupProgram.bind(plan, weights, x, gain)
    for _ in range(2):       # the counters are clean for the second
        program.submit_for_plan()
        ctx["stream"].synchronize()
        assert plan.device_status() == 0
        staged = bits_from_torch_bf16(program.staged)
        for out, r, planes in zip(program.outputs, rows, made):
            y64 = oracle.linear_f64(*planes, r, cols, staged, threads=oracle.max_threads())
            assert rel_error(bits_from_torch_bf16(out), y64.reshape(tokens, r)) <= TOLERANCE
    plan.close()
