"""How the pair GEMM shares main and tail tiles out between pairs of CTAs, on the host (tests/cpp/pair_work_test.cpp) with the headers that
the library includes: 20000 random launches and those chosen for 20000 random GEMMs, every part of every tile done once and handed over to the
pair that waits for it; and that the GPU tests of tail tiles and leftover tiles take the path that they are there for."""
import pathlib
import subprocess

import pytest

from test_gpu_prefill_tails import BLOCKS, CASES, LEFTOVER, LEFTOVER_BLOCKS
from test_gpu_prefill_token_ranges import NARROW

ROOT = pathlib.Path(__file__).resolve().parents[1]
PAIRS = 74      # of CTAs on a B200: as many slots has a plan with room to cut tiles


@pytest.fixture(scope="module")
def binary(tmp_path_factory):
    path = tmp_path_factory.mktemp("pair_work") / "pair_work_test"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "augur_v100_b200/csrc"), "-o", str(path), str(ROOT / "tests/cpp/pair_work_test.cpp")],
                   check=True, capture_output=True, text=True, timeout=120)
    return path


def test_every_part_of_every_tile_once(binary):
    done = subprocess.run([str(binary)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0 and done.stdout.strip() == "ok", done.stdout


def _chosen(binary, rows, cols, tokens, terms, gate_up, slots, pairs=False):
    done = subprocess.run([str(binary)] + [str(v) for v in (rows, cols, tokens, terms, gate_up, slots)], capture_output=True, text=True, timeout=60, check=True)
    token_pairs, tail_columns, sharers, given, finished = map(int, done.stdout.split())
    if pairs:
        return token_pairs
    return tail_columns, given > 0 and finished > 0, sharers


@pytest.mark.parametrize("rows,cols,tokens,terms,tail,cut,tail_without", CASES)
def test_tail_cases(binary, rows, cols, tokens, terms, tail, cut, tail_without):
    assert _chosen(binary, rows, cols, tokens, terms, 0, PAIRS)[:2] == (tail, cut)
    assert _chosen(binary, rows, cols, tokens, terms, 0, 0) == (tail_without, False, 0)


@pytest.mark.parametrize("hidden,inter,tokens,terms,tail,cut", BLOCKS)
def test_tail_blocks(binary, hidden, inter, tokens, terms, tail, cut):
    assert _chosen(binary, 2 * inter, hidden, tokens, terms, 1, PAIRS)[:2] == (tail, cut)


@pytest.mark.parametrize("rows,cols,tokens,terms,sharers", LEFTOVER)
def test_leftover_cases(binary, rows, cols, tokens, terms, sharers):
    assert _chosen(binary, rows, cols, tokens, terms, 0, PAIRS) == (0, False, sharers)


@pytest.mark.parametrize("hidden,inter,tokens,terms,sharers", LEFTOVER_BLOCKS)
def test_leftover_blocks(binary, hidden, inter, tokens, terms, sharers):
    assert _chosen(binary, 2 * inter, hidden, tokens, terms, 1, PAIRS) == (0, False, sharers)


@pytest.mark.parametrize("rows,cols,tokens,terms", NARROW + [(128, 64, 9, 1), (384, 192, 16, 3), (128, 320, 17, 2), (2944, 2112, 127, 3), (640, 1088, 129, 3),
                                                             (128, 17408, 33, 2)])
def test_narrow_cases(binary, rows, cols, tokens, terms):
    assert _chosen(binary, rows, cols, tokens, terms, 0, PAIRS, pairs=True) == 0
    assert _chosen(binary, rows, cols, tokens, terms, 0, 0, pairs=True) == 0


# The choice between the two kernels. us by the narrow one and by pairs: an estimate fitted to 130 tokens and more had taken the slower of them.
@pytest.mark.parametrize("rows,cols,tokens,terms,gate_up,narrow", [
    (9600, 64, 15, 1, 0, True),         # 4.3 / 6.5
    (14464, 1792, 69, 2, 0, True),      # 10.3 / 11.3
    (18944, 1088, 160, 3, 1, True),     # 18.3 / 24.1
    (7424, 1024, 450, 2, 1, True),      # 13.7 / 18.1
    (2048, 1792, 1669, 1, 1, True),     # 13.3 / 18.6
    (33536, 1024, 1402, 2, 1, False)])  # 105 / 89
def test_quicker_kernel(binary, rows, cols, tokens, terms, gate_up, narrow):
    assert (_chosen(binary, rows, cols, tokens, terms, gate_up, PAIRS, pairs=True) == 0) is narrow


# GEMMs that a cut cost more than it saved, or that went to tail tiles whose quantiser takes longer than their k blocks: us as chosen here and as by a rule that took
# a cut for hidden under whole tiles and shares of two tiles for as good as even ones.
@pytest.mark.parametrize("rows,cols,tokens,terms,gate_up,most", [
    (1536, 6016, 3776, 1, 0, 32),       # 27.5 / 32.8 by 74 pairs
    (5376, 4864, 2773, 3, 0, 45),       # 113 / 120 by 72
    (5376, 4864, 2773, 1, 0, 0),        # 52 / 57 by 36
    (3456, 7552, 1761, 3, 0, 72),       # 83.2 / 84.8 by 74
    (2560, 3456, 2412, 1, 1, 0),        # 23.6 / 35.4 by 73
    (5120, 1408, 810, 2, 1, 0),         # 13.0 / 22.0 with tail tiles
    (10496, 1152, 301, 3, 1, 0)])       # 18.2 / 32.3 with tail tiles
def test_cuts_that_cost_more(binary, rows, cols, tokens, terms, gate_up, most):
    tail_columns, _, sharers = _chosen(binary, rows, cols, tokens, terms, gate_up, PAIRS)
    assert tail_columns == 0 and sharers <= most
