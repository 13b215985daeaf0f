"""How the pair GEMM shares main and tail tiles out between pairs of CTAs, on the host (tests/cpp/pair_work_test.cpp) with the headers that
the library includes: 20000 random launches and those chosen for 20000 random GEMMs, every part of every tile done once and handed over to the
pair that waits for it; and that the GPU tests of the tail tiles take the path that they are there for."""
import pathlib
import subprocess

import pytest

from test_gpu_prefill_tails import BLOCKS, CASES

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


def _chosen(binary, rows, cols, tokens, terms, slots):
    done = subprocess.run([str(binary)] + [str(v) for v in (rows, cols, tokens, terms, slots)], capture_output=True, text=True, timeout=60, check=True)
    _, tail_columns, _, given, finished = map(int, done.stdout.split())
    return tail_columns, given > 0 and finished > 0


@pytest.mark.parametrize("rows,cols,tokens,terms,tail,cut,tail_without", CASES)
def test_tail_cases(binary, rows, cols, tokens, terms, tail, cut, tail_without):
    assert _chosen(binary, rows, cols, tokens, terms, PAIRS) == (tail, cut)
    assert _chosen(binary, rows, cols, tokens, terms, 0) == (tail_without, False)


@pytest.mark.parametrize("hidden,inter,tokens,terms,tail,cut", BLOCKS)
def test_tail_blocks(binary, hidden, inter, tokens, terms, tail, cut):
    assert _chosen(binary, 2 * inter, hidden, tokens, terms, PAIRS) == (tail, cut)
