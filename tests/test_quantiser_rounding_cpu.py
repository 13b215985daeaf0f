"""The two shortcuts of the quantiser's rounding against the rules they stand for, on the host (tests/cpp/rounding_test.cpp), with the
constant and the steps of the header that the kernels include: E2M1 ties for every F32 quotient from 2^-6 to 16 and a share of
all others, the block scale's quotient for 2 * 10^7 pairs. Exact: any difference fails."""
import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_ties_and_block_scale_quotients(tmp_path):
    binary = tmp_path / "rounding_test"
    # no contraction: a product and a sum that the source keeps apart stay two roundings, as in the kernels
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "augur_v100_b200/csrc"), "-o", str(binary),
                    str(ROOT / "tests/cpp/rounding_test.cpp")], check=True, capture_output=True, text=True, timeout=120)
    done = subprocess.run([str(binary)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0 and done.stdout.strip() == "ok", done.stdout
