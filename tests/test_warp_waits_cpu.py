"""Bounded waits of the tensor-memory kernels, read from their source.

A warp that issues tcgen05 or TMA operations elects a lane for them, and an election, like a shuffle or a tensor-memory load, needs
all 32 lanes. Lanes that poll a barrier need not see the same of it, so a lane whose wait failed must not leave its warp alone: code
of a whole warp uses the waits that give all lanes the same answer (warp_wait and its forms); mbar_wait, which does not, is for roles
of one lane, or where nothing is decided on its result. And what a worker of the one-launch block decides alone must not take it out of the loop in which the workers meet."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "augur_v100_b200" / "csrc"
FILES = ["bf16_head.cu", "nvfp4_gemm.cu", "nvfp4_gemm_narrow.cu", "nvfp4_gemv_split.cu", "nvfp4_gemv_tc.cu"]


def source(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def blocks_around(text, at):
    """Headers of the blocks around a position, outermost first."""
    blocks, start, parentheses = [], 0, 0
    for i, char in enumerate(text[:at]):
        parentheses += (char == "(") - (char == ")")
        if char in "{}" or (char == ";" and not parentheses):
            if char == "{":
                blocks.append(" ".join(text[start:i].split()))
            elif char == "}":
                blocks.pop()
            start = i + 1
    return blocks


@pytest.mark.parametrize("name", FILES)
def test_a_wait_of_one_lane_is_used_by_roles_of_one_lane(name):
    text = source(name)
    assert re.search(r"\bwarp_(?:look_)?wait\(", text)
    for found in re.finditer(r"\bmbar_wait\w*\(", text):
        unused = text[:found.start()].rstrip()[-1] in ";{}"   # nothing is decided on it
        assert unused or any("lane == 0" in header for header in blocks_around(text, found.start())), text[found.start():found.start() + 80]


@pytest.mark.parametrize("name", FILES)
def test_there_is_a_counter_for_every_warp_that_waits(name):
    """Where a failed wait's lanes meet: behind the abort flag, cleared with it."""
    text = source(name)
    assert text.count("*abort_flag = 0;") == 1
    assert re.search(r"\*abort_flag = 0;\s*for \(uint32_t w = 0; w < (?:k\w*Threads / 32|kSmallStateWarps); \+\+w\) abort_flag\[1 \+ w\] = 0;", text)


def test_workers_stay_in_step():
    text = source("nvfp4_gemv_tc.cu")
    start = text.index("for (uint32_t s = 0; s < p.steps; ++s)")
    loop = text[start:text.index("p.header[kHeaderEpoch] = meeting;")]
    # the only breaks are those of polls
    for found in re.finditer(r"\bbreak;", loop):
        assert any(header.startswith("for (uint32_t spin = 0;") for header in blocks_around(text, start + found.start())), loop[:found.start()][-120:]
    assert "return" not in loop
