"""A repack and the launch behind it on one stream, without a synchronise between them: through the C ABI a submit only enqueues,
and stream order is all that a caller has. Every consumer that fetches weights early is here, with the destination holding other
valid weights, so that a stale block shows; results equal those of the synchronised order bit for bit."""
from ctypes import byref, c_uint64

import pytest

from augur_v100_b200 import abi, host, synth

pytestmark = pytest.mark.gpu

ROWS, COLS = 8192, 4096


@pytest.fixture(scope="module")
def env():
    import torch
    torch.cuda.set_device(0)
    side = torch.cuda.Stream()
    stream = host.Stream(0, side)
    plan = host.Plan(stream, 64 << 20)
    generator = torch.Generator(device="cuda")
    generator.manual_seed(11)
    planes = []
    for _ in range(2):
        scales = (torch.randn((ROWS, COLS // 16), device="cuda", generator=generator).abs() * 0.5).clamp(2.0 ** -9, 448.0)
        planes.append((torch.randint(0, 256, (ROWS, COLS // 2), dtype=torch.uint8, device="cuda", generator=generator),
                       scales.to(torch.float8_e4m3fn).view(torch.uint8).clamp(1, 0x7E)))
    torch.cuda.synchronize()
    yield {"torch": torch, "side": side, "stream": stream, "plan": plan, "planes": planes}
    plan.close()
    stream.close()


def _repack_args(weight, planes, rows=ROWS, cols=COLS):
    args = abi.header(abi.RepackArgs)
    for name, tensor in (("codes", planes[0]), ("scales", planes[1]), ("destination", weight.packed)):
        setattr(args, name, tensor.data_ptr())
        setattr(args, name + "_len_bytes", tensor.numel())
    args.rows, args.cols, args.layout = rows, cols, weight.layout
    return args


# one launch on mma.sync; one on tensor memory; two, and quantiser and narrow GEMM, whose weights are fetched behind a launch that triggers early;
# pair GEMM
@pytest.mark.parametrize("kind,tokens,rows,cols,launches", [("stream", 3, ROWS, COLS, 1), ("split", 8, ROWS, COLS, 1), ("split", 8, 1024, 8 * COLS, 2),
                                                            ("gemm", 16, ROWS, COLS, 2), ("gemm", 300, ROWS, COLS, 2)])
def test_repack_then_linear(env, kind, tokens, rows, cols, launches):
    torch, side, stream, plan = env["torch"], env["side"], env["stream"], env["plan"]
    planes = [(codes.view(rows, cols // 2), scales.view(rows, cols // 16)) for codes, scales in env["planes"]]
    layout = abi.LAYOUT_STREAM if kind == "stream" else abi.LAYOUT_TCGEN05
    with torch.cuda.stream(side):
        generator = torch.Generator(device="cuda")
        generator.manual_seed(tokens)
        x = torch.randn((tokens, cols), device="cuda", generator=generator).to(torch.bfloat16)
        weight = host.Nvfp4Sm100Weight.repack_device_planes(stream, layout, rows, cols, *planes[0], synth.GLOBAL_SCALE)
        binding = {"stream": host.Nvfp4Sm100Projection, "split": host.Nvfp4Sm100TcProjection, "gemm": host.Nvfp4Sm100PrefillLinear}[kind]
        program = binding.bind(plan, weight, x)
        submit = abi.lib().augur_cuda_nvfp4_sm100_repack_prevalidated_submit_v1
        args = [_repack_args(weight, both, rows, cols) for both in planes]
        wanted = []
        for which in range(2):
            assert submit(stream.ordinal, stream.handle, byref(args[which])).status == abi.STATUS_OK
            stream.synchronize()
            before = host.launch_count()
            program.submit_for_plan()
            assert host.launch_count() - before == launches
            stream.synchronize()
            wanted.append(program.out.clone())
        got = []
        for turn in range(40):
            assert submit(stream.ordinal, stream.handle, byref(args[turn % 2])).status == abi.STATUS_OK
            program.submit_for_plan()
            got.append(program.out.clone())
        side.synchronize()
    assert plan.device_status() == 0
    assert not torch.equal(wanted[0], wanted[1])
    assert [torch.equal(out, wanted[turn % 2]) for turn, out in enumerate(got)] == [True] * 40


# The quantiser reads what the launch before it writes, while that launch still runs: narrow GEMM, pair GEMM, small-token
# linear on tensor memory.
@pytest.mark.parametrize("tokens,producer", [(48, "gemm"), (300, "gemm"), (8, "split")])
def test_linear_then_quantiser(env, tokens, producer):
    torch, side, stream, plan = env["torch"], env["side"], env["stream"], env["plan"]
    with torch.cuda.stream(side):
        generator = torch.Generator(device="cuda")
        generator.manual_seed(tokens)
        inputs = [torch.randn((tokens, COLS), device="cuda", generator=generator).to(torch.bfloat16) for _ in range(2)]
        x = inputs[0].clone()
        weight = host.Nvfp4Sm100Weight.repack_device_planes(stream, abi.LAYOUT_TCGEN05, ROWS, COLS, *env["planes"][0], synth.GLOBAL_SCALE)
        second = host.Nvfp4Sm100Weight.repack_device_planes(
            stream, abi.LAYOUT_TCGEN05, COLS, ROWS, env["planes"][1][0].view(COLS, ROWS // 2), env["planes"][1][1].view(COLS, ROWS // 16), synth.GLOBAL_SCALE)
        first = {"gemm": host.Nvfp4Sm100PrefillLinear, "split": host.Nvfp4Sm100TcProjection}[producer].bind(plan, weight, x)
        then = host.Nvfp4Sm100PrefillLinear.bind(plan, second, first.out, terms=3)
        wanted = []
        for value in inputs:
            x.copy_(value)
            first.submit_for_plan()
            stream.synchronize()
            then.submit_for_plan()
            stream.synchronize()
            wanted.append(then.out.clone())
        got = []
        for turn in range(40):
            x.copy_(inputs[turn % 2])
            first.submit_for_plan()
            then.submit_for_plan()
            got.append(then.out.clone())
        side.synchronize()
    assert plan.device_status() == 0
    assert not torch.equal(wanted[0], wanted[1])
    assert [torch.equal(out, wanted[turn % 2]) for turn, out in enumerate(got)] == [True] * 40


def _lagging_launch(env, plan):
    """A tensor-parallel launch of a few CTAs whose peer never answers: it lets its successors start at once and gives up after
    about a second (bounded polls). What it reads and writes is returned, to be kept."""
    torch, stream = env["torch"], env["stream"]
    hidden, inter, tokens, world = 128, 256, 8, 2
    weights = [host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(stream, abi.LAYOUT_STREAM_PAIR, inter, hidden, *synth.make_weight(3, 98, "gate", inter, hidden),
                                                             *synth.make_weight(3, 98, "up", inter, hidden)),
               host.Nvfp4Sm100Weight.upload_checkpoint_nvfp4(stream, abi.LAYOUT_STREAM, hidden, inter, *synth.make_weight(3, 98, "down", hidden, inter))]
    program = host.Nvfp4Sm100FfnProgram.bind(plan, *weights, torch.ones((tokens, hidden), dtype=torch.bfloat16, device="cuda"))
    extent = c_uint64()
    assert abi.lib().augur_cuda_nvfp4_sm100_mlp_tp_exchange_extent_host_v1(hidden, world, byref(extent)).status == abi.STATUS_OK
    buffers = [torch.zeros(extent.value, dtype=torch.uint8, device="cuda") for _ in range(world)]
    args = abi.header(abi.MlpTpArgs)
    args.gate_up, args.down = program.args.gate_up, program.args.down
    for rank, buffer in enumerate(buffers):
        args.exchange[rank] = buffer.data_ptr()
    args.exchange_len_bytes, args.world, args.rank, args.sequence = extent.value, world, 0, 1
    torch.cuda.synchronize()
    submit = abi.lib().augur_cuda_nvfp4_sm100_mlp_tp_prevalidated_submit_v1
    assert submit(stream.ordinal, stream.handle, plan.handle, byref(args)).status == abi.STATUS_OK
    return program, buffers


# The bounded waits of a launch do not run out while it waits for a launch ahead of it that takes long: small-token linear of one launch and of
# two, narrow GEMM, pair GEMM, one-launch MLP block.
@pytest.mark.parametrize("kind,tokens,rows,cols", [("split", 8, ROWS, COLS), ("split", 8, 1024, 8 * COLS), ("gemm", 16, ROWS, COLS), ("gemm", 300, ROWS, COLS),
                                                   ("block", 8, ROWS, COLS)])
def test_waits_do_not_count_the_launch_before(env, kind, tokens, rows, cols):
    torch, side, stream, plan = env["torch"], env["side"], env["stream"], env["plan"]
    with torch.cuda.stream(side):
        x = torch.randn((tokens, cols), device="cuda").to(torch.bfloat16)
        codes, scales = env["planes"][0]
        weight = host.Nvfp4Sm100Weight.repack_device_planes(stream, abi.LAYOUT_TCGEN05, rows, cols, codes.view(rows, cols // 2), scales.view(rows, cols // 16),
                                                            synth.GLOBAL_SCALE)
        if kind == "block":
            weight.global_scale_b = synth.GLOBAL_SCALE   # the rows as gate and up of an intermediate half as wide
            codes, scales = (plane[:COLS] for plane in env["planes"][1])
            down = host.Nvfp4Sm100Weight.repack_device_planes(stream, abi.LAYOUT_TCGEN05, COLS, ROWS // 2, codes, scales, synth.GLOBAL_SCALE)
            program = host.Nvfp4Sm100TcFfnProgram.bind(plan, weight, down, x)
        else:
            program = {"split": host.Nvfp4Sm100TcProjection, "gemm": host.Nvfp4Sm100PrefillLinear}[kind].bind(plan, weight, x)
        program.submit_for_plan()
        wanted = program.out.clone()
        program.out.zero_()
        lagging = host.Plan(stream, host.mlp_scratch_bytes(128, 256))
        kept = _lagging_launch(env, lagging)
        program.submit_for_plan()
        stream.synchronize()
    assert lagging.device_status() == 0x203 and plan.device_status() == 0
    assert torch.equal(program.out, wanted)
    del kept
    lagging.close()


# The head's weights are any BF16 matrix: here the output of a linear that lets its successor start before it has stored anything,
# with other values in the buffer; and the head behind a launch that takes long.
def test_head_behind_the_launch_that_writes_its_weight(env):
    torch, side, stream, plan = env["torch"], env["side"], env["stream"], env["plan"]
    tokens = 48
    with torch.cuda.stream(side):
        x = torch.randn((tokens, COLS), device="cuda").to(torch.bfloat16)
        weight = host.Nvfp4Sm100Weight.repack_device_planes(stream, abi.LAYOUT_TCGEN05, ROWS, COLS, *env["planes"][0], synth.GLOBAL_SCALE)
        producer = host.Nvfp4Sm100PrefillLinear.bind(plan, weight, x)
        head = host.Bf16Head.bind(stream, producer.out.view(2 * tokens, ROWS // 2), torch.randn((4, ROWS // 2), device="cuda"))
        producer.submit_for_plan()
        stream.synchronize()
        head.submit()
        wanted = head.out.clone()
        got = []
        for _ in range(20):
            producer.out.zero_()
            producer.submit_for_plan()
            head.submit()
            got.append(head.out.clone())
        lagging = host.Plan(stream, host.mlp_scratch_bytes(128, 256))
        kept = _lagging_launch(env, lagging)
        head.submit()
        got.append(head.out.clone())
        stream.synchronize()
    assert lagging.device_status() == 0x203 and plan.device_status() == 0
    assert [torch.equal(out, wanted) for out in got] == [True] * 21
    del kept
    lagging.close()
