"""How the pair GEMM shares main and tail tiles out between pairs of CTAs, on the host (tests/cpp/pair_work_test.cpp) with the header that
the kernel includes: 20000 random launches, every part of every tile done once and handed over to the pair that waits for it."""
import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_every_part_of_every_tile_once(tmp_path):
    binary = tmp_path / "pair_work_test"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "augur_v100_b200/csrc"), "-o", str(binary), str(ROOT / "tests/cpp/pair_work_test.cpp")],
                   check=True, capture_output=True, text=True, timeout=120)
    done = subprocess.run([str(binary)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0 and done.stdout.strip() == "ok", done.stdout
