"""What this library's speed is measured on: the calls a model runtime makes, through the public host classes.

Kinds of work, each a range of which `listed()` names the points that real use meets most and `draw()` gives more:

  linear      one quantised weight behind `Nvfp4Sm100Linear`, the dispatch a runtime keeps per call site: decode and
              verify batches of 1..8 token rows, prompts and batched decode of any wider count up to a 4096-row chunk
              (`terms` = 3: BF16-accurate activations, the default; 2 or 1: FP4 activations).
  block       the MLP block: the one-launch program or the two-launch program (`program`) up to 8 token rows, the
              prefill program beyond.
  layers      a verify pass over whole layers, each three attention-side projections and the MLP block, every launch
              behind the one before it, as the decode loop of a model issues them.
  norm_group  residual add, RMSNorm and the projections that share the normalised input.
  head        the BF16 vocabulary head.
  load        a checkpoint weight brought into both hot layouts.

Weights are uniform E2M1 codes with E4M3 block scales |N(0,1)| * 0.5 and the tensor scale 1/448, activations N(0,1) in
BF16: the distributions of the benchmark configurations. Everything runs on one stream of its own, as in a serving
loop. Three states in rotation hold more than the L2 cache for all but the small shards, whose weights are also
warm in real use when one layer is called again.
"""
import math

import torch

from augur_v100_b200 import abi, host, synth

HIDDEN, INTERMEDIATE, VOCABULARY = 5120, 17408, 248320
WEIGHT_BYTES = 9.0 / 16.0          # 4-bit code and a sixteenth of an 8-bit scale, per weight

_side = None


def _stream():
    """The serving loop's stream, one for the life of the program."""
    global _side
    if _side is None:
        side = torch.cuda.Stream()
        _side = (side, host.Stream(torch.cuda.current_device(), side))
    return _side


def listed():
    return [
        # a key or value projection while one user decodes: the smallest call, all latency
        {"name": "linear 1024x5120 m1", "kind": "linear", "rows": 1024, "cols": 5120, "tokens": 1, "terms": 3},
        # one up-type projection at the speculative-verify batch
        {"name": "linear 17408x5120 m8", "kind": "linear", "rows": 17408, "cols": 5120, "tokens": 8, "terms": 3},
        # a short prompt, or 48 users decoding together
        {"name": "linear 6144x5120 m48", "kind": "linear", "rows": 6144, "cols": 5120, "tokens": 48, "terms": 3},
        # a full prefill chunk, FP4 activations
        {"name": "linear 17408x5120 m4096", "kind": "linear", "rows": 17408, "cols": 5120, "tokens": 4096, "terms": 1},
        # the MLP block of the 27B-class model at the verify batch
        {"name": "block m8", "kind": "block", "hidden": HIDDEN, "inter": INTERMEDIATE, "tokens": 8, "terms": 3, "program": "one launch"},
        # one rank's shard of it (8-way tensor-parallel width) for a single decoded token, on the program that shards use
        {"name": "block shard m1", "kind": "block", "hidden": HIDDEN, "inter": INTERMEDIATE // 8, "tokens": 1, "terms": 3, "program": "two launches"},
        # a ragged prompt
        {"name": "block m777", "kind": "block", "hidden": HIDDEN, "inter": INTERMEDIATE, "tokens": 777, "terms": 3, "program": "prefill"},
        # a full prefill chunk at BF16-activation accuracy: the largest call
        {"name": "block m4096", "kind": "block", "hidden": HIDDEN, "inter": INTERMEDIATE, "tokens": 4096, "terms": 3, "program": "prefill"},
        # two layers of a verify pass
        {"name": "layers m8", "kind": "layers", "count": 2, "hidden": HIDDEN, "inter": INTERMEDIATE, "wide": 10240, "tokens": 8},
        # the input group of a gated-delta-net layer, gates of 48 rows among its members
        {"name": "norm group m8", "kind": "norm_group", "cols": HIDDEN, "rows_a": 10240, "rows_b": 6144, "gates": 2, "residual": True, "tokens": 8},
        # the vocabulary head at the verify batch
        {"name": "head m8", "kind": "head", "rows": VOCABULARY, "cols": HIDDEN, "tokens": 8},
        # loading one up-type projection for both batch classes
        {"name": "load 17408x5120", "kind": "load", "rows": INTERMEDIATE, "cols": HIDDEN},
    ]


def _spread(rng, low, high, step):
    """A multiple of `step` in [low, high], even over the logarithm."""
    return min(high // step, max(-(-low // step), round(math.exp(rng.uniform(math.log(low), math.log(high))) / step))) * step


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "block", "block", "block", "layers", "norm_group", "head", "load"])
    small = rng.randint(1, abi.MAX_SMALL_TOKENS)
    tokens = small if rng.random() < 0.4 else _spread(rng, abi.MAX_SMALL_TOKENS + 1, 4096, 1)
    terms = rng.choice([3, 3, 2, 1])
    if kind == "linear" or kind == "load":
        sides = [_spread(rng, 1024, 10240, 128), _spread(rng, 1024, INTERMEDIATE, 128)]
        rng.shuffle(sides)
        case = {"kind": kind, "rows": sides[0], "cols": sides[1]}
        return case if kind == "load" else dict(case, tokens=tokens, terms=terms)
    if kind == "block":
        program = "prefill" if tokens > abi.MAX_SMALL_TOKENS else rng.choice(["one launch", "two launches"])
        return {"kind": kind, "hidden": _spread(rng, 1024, HIDDEN, 128), "inter": _spread(rng, 1024, INTERMEDIATE, 128),
                "tokens": tokens, "terms": terms, "program": program}
    if kind == "layers":
        return {"kind": kind, "count": rng.randint(1, 2), "hidden": _spread(rng, 1024, HIDDEN, 128),
                "inter": _spread(rng, 2048, INTERMEDIATE, 128), "wide": _spread(rng, 1024, 10240, 128), "tokens": small}
    if kind == "norm_group":
        return {"kind": kind, "cols": _spread(rng, 1024, HIDDEN, 256), "rows_a": _spread(rng, 1024, 12288, 32),
                "rows_b": _spread(rng, 1024, 6144, 32), "gates": rng.randint(0, 2), "residual": rng.random() < 0.5, "tokens": small}
    return {"kind": "head", "rows": _spread(rng, 32000, VOCABULARY, 16), "cols": _spread(rng, 1024, HIDDEN, 64), "tokens": small}


# ---- what a program holds before the call ------------------------------------------------------------------
def _planes(generator, rows, cols):
    """Checkpoint planes of one weight: packed codes and block scales."""
    device = generator.device
    codes = torch.randint(0, 256, (rows, cols // 2), dtype=torch.uint8, device=device, generator=generator)
    raw = (torch.randn((rows, cols // 16), device=device, generator=generator).abs() * 0.5).clamp(2.0 ** -9, 448.0)
    return codes, raw.to(torch.float8_e4m3fn).view(torch.uint8).clamp(1, 0x7E)


def _weight(stream, generator, layout, rows, cols):
    codes, scales = _planes(generator, rows, cols)
    return host.Nvfp4Sm100Weight.repack_device_planes(stream, layout, rows, cols, codes, scales, synth.GLOBAL_SCALE)


def _gate_up(stream, generator, inter, hidden):
    """The gate and up matrices as one tcgen05 weight, 16 gate rows alternating with the matching 16 up rows."""
    planes = [torch.stack([gate.view(inter // 16, 16, -1), up.view(inter // 16, 16, -1)], dim=1).reshape(2 * inter, -1).contiguous()
              for gate, up in zip(_planes(generator, inter, hidden), _planes(generator, inter, hidden))]
    weight = host.Nvfp4Sm100Weight.repack_device_planes(stream, abi.LAYOUT_TCGEN05, 2 * inter, hidden, *planes, synth.GLOBAL_SCALE)
    weight.global_scale_b = synth.GLOBAL_SCALE
    return weight


def _activations(generator, tokens, cols):
    return torch.randn((tokens, cols), device=generator.device, generator=generator).to(torch.bfloat16)


def _prepare_linear(case, stream, generator):
    rows, cols, tokens = case["rows"], case["cols"], case["tokens"]
    codes, scales = (plane.cpu().numpy() for plane in _planes(generator, rows, cols))
    linear = host.Nvfp4Sm100Linear(stream, rows, cols, codes, scales, synth.GLOBAL_SCALE)
    plan = host.Plan(stream, max(host.gemm_plan_scratch_bytes(), host.gemv_scratch_bytes(rows, cols)))
    return {"program": linear.bind(plan, _activations(generator, tokens, cols), terms=case["terms"]), "linear": linear, "plan": plan}


def _prepare_block(case, stream, generator):
    hidden, inter, tokens = case["hidden"], case["inter"], case["tokens"]
    x = _activations(generator, tokens, hidden)
    if case["program"] == "two launches":
        gate_up = host.Nvfp4Sm100Weight.repack_device_planes(
            stream, abi.LAYOUT_STREAM_PAIR, inter, hidden, *_planes(generator, inter, hidden), synth.GLOBAL_SCALE,
            *_planes(generator, inter, hidden), synth.GLOBAL_SCALE)
        down = _weight(stream, generator, abi.LAYOUT_STREAM, hidden, inter)
        plan = host.Plan(stream, host.mlp_scratch_bytes(hidden, inter))
        return {"program": host.Nvfp4Sm100FfnProgram.bind(plan, gate_up, down, x), "plan": plan}
    gate_up = _gate_up(stream, generator, inter, hidden)
    down = _weight(stream, generator, abi.LAYOUT_TCGEN05, hidden, inter)
    if case["program"] == "one launch":
        plan = host.Plan(stream, host.mlp_tc_scratch_bytes(hidden, inter))
        return {"program": host.Nvfp4Sm100TcFfnProgram.bind(plan, gate_up, down, x), "plan": plan}
    plan = host.Plan(stream, host.gemm_plan_scratch_bytes())
    program = host.Nvfp4Sm100PrefillFfnProgram.bind(plan, gate_up, down, x, terms=case["terms"], intermediate_global_scale=2.0 ** -6)
    return {"program": program, "plan": plan}


def _prepare_layers(case, stream, generator):
    hidden, inter, wide, tokens = case["hidden"], case["inter"], case["wide"], case["tokens"]
    shapes = ((wide, hidden), (hidden, hidden), (hidden, wide))
    plan = host.Plan(stream, max([host.mlp_tc_scratch_bytes(hidden, inter)] + [host.gemv_tc_scratch_bytes(r, c) for r, c in shapes]))
    x = _activations(generator, tokens, hidden)
    members = []
    for _ in range(case["count"]):
        # the attention or delta-net core between the projections is not this library's: its output is an input here
        mixed = _activations(generator, tokens, wide)
        inputs = (x, x, mixed)
        projections = [host.Nvfp4Sm100TcProjection.bind(plan, _weight(stream, generator, abi.LAYOUT_TCGEN05, r, c), value)
                       for (r, c), value in zip(shapes, inputs)]
        block = host.Nvfp4Sm100TcFfnProgram.bind(plan, _gate_up(stream, generator, inter, hidden),
                                                 _weight(stream, generator, abi.LAYOUT_TCGEN05, hidden, inter), projections[2].out)
        members += projections + [block]
        x = block.out
    return {"members": members, "plan": plan}


def _prepare_norm_group(case, stream, generator):
    cols, tokens, device = case["cols"], case["tokens"], generator.device
    rows = [case["rows_a"], case["rows_b"]] + [64] * case["gates"]
    weights = [_weight(stream, generator, abi.LAYOUT_STREAM, r, cols) for r in rows]
    norm_weight = 1.0 + 0.1 * torch.randn((cols,), device=device, generator=generator)
    residual, update = (2.0 * torch.randn((tokens, cols), device=device, generator=generator) for _ in range(2))
    plan = host.Plan(stream, 64 << 20)
    adds = (torch.empty_like(residual), residual, update) if case["residual"] else (residual, None, None)
    program = host.Nvfp4Sm100NormGroupProgram.bind(plan, weights, adds[0], norm_weight, add_a=adds[1], add_b=adds[2],
                                                   stored_rows=[0, 0] + [48] * case["gates"])
    return {"program": program, "plan": plan}


def _prepare_head(case, stream, generator):
    weight = torch.empty((case["rows"], case["cols"]), dtype=torch.bfloat16, device=generator.device).normal_(0.0, 0.02, generator=generator)
    x = torch.randn((case["tokens"], case["cols"]), device=generator.device, generator=generator)
    return {"program": host.Bf16Head.bind(stream, weight, x)}


def _prepare_load(case, stream, generator):
    return {"planes": _planes(generator, case["rows"], case["cols"])}


_PREPARE = {"linear": _prepare_linear, "block": _prepare_block, "layers": _prepare_layers, "norm_group": _prepare_norm_group,
            "head": _prepare_head, "load": _prepare_load}


def prepare(case, seed):
    side, stream = _stream()
    with torch.cuda.stream(side):
        generator = torch.Generator(device=torch.device("cuda", torch.cuda.current_device()))
        generator.manual_seed(seed)
        state = _PREPARE[case["kind"]](case, stream, generator)
    state.update(case=case, side=side, stream=stream)
    return state


# ---- one pass ----------------------------------------------------------------------------------------------
def run(state):
    kind = state["case"]["kind"]
    if kind == "load":
        rows, cols, (codes, scales) = state["case"]["rows"], state["case"]["cols"], state["planes"]
        with torch.cuda.stream(state["side"]):
            return [host.Nvfp4Sm100Weight.repack_device_planes(state["stream"], layout, rows, cols, codes, scales, synth.GLOBAL_SCALE).packed
                    for layout in (abi.LAYOUT_STREAM, abi.LAYOUT_TCGEN05)]
    if kind == "layers":
        for member in state["members"]:
            member.submit_for_plan()
        return [member.out for member in state["members"]]
    program = state["program"]
    if kind == "head":
        program.submit()
        return program.out
    program.submit_for_plan()
    if kind == "norm_group":
        return [program.input, program.normalised, program.staged] + program.outputs
    if kind == "block" and state["case"]["program"] != "prefill":
        return [program.intermediate, program.out]
    return program.out


# ---- what a pass cannot do without ---------------------------------------------------------------------------
def _linear_work(rows, cols, tokens):
    return rows * cols * WEIGHT_BYTES + tokens * (cols + rows) * 2.0, 2.0 * tokens * rows * cols


def _block_work(hidden, inter, tokens):
    return 3.0 * hidden * inter * WEIGHT_BYTES + tokens * hidden * 4.0, 6.0 * tokens * hidden * inter


def work(case):
    kind, tokens = case["kind"], case.get("tokens", 0)
    if kind == "linear":
        parts = [_linear_work(case["rows"], case["cols"], tokens)]
    elif kind == "block":
        parts = [_block_work(case["hidden"], case["inter"], tokens)]
    elif kind == "layers":
        hidden, wide = case["hidden"], case["wide"]
        parts = [_linear_work(wide, hidden, tokens), _linear_work(hidden, hidden, tokens), _linear_work(hidden, wide, tokens),
                 _block_work(hidden, case["inter"], tokens)] * case["count"]
    elif kind == "norm_group":
        # residual operands in, their sum and the normalised rows out (F32), the norm weight; the members read the BF16 rows
        parts = [(tokens * case["cols"] * 4.0 * (4 if case["residual"] else 2) + case["cols"] * 4.0, 0.0)]
        parts += [_linear_work(r, case["cols"], tokens) for r in (case["rows_a"], case["rows_b"]) + (48,) * case["gates"]]
    elif kind == "head":
        rows, cols = case["rows"], case["cols"]
        parts = [(rows * cols * 2.0 + tokens * (rows + cols) * 4.0, 2.0 * tokens * rows * cols)]
    else:
        # the planes in once, each of the two layouts out
        parts = [(3.0 * case["rows"] * case["cols"] * WEIGHT_BYTES, 0.0)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    if case["kind"] == "load":
        return "exact"
    if case["kind"] == "head":
        return {"rel": 1e-5}
    # BF16 results; where activations are quantised the levels are fixed by rule, so only sums and roundings may differ
    return {"rel": 1e-2, "max": 5e-2}
