"""Which small-token kernel `Nvfp4Sm100Linear` takes below the line of the large weights: a rule on rows, columns, token rows and scratch."""
from types import SimpleNamespace

import pytest

from augur_v100_b200 import host


@pytest.mark.parametrize("rows,cols,tokens,expected", [
    (1024, 5120, 1, True), (1024, 5120, 4, True), (1024, 5120, 5, True), (1024, 5120, 6, False), (1024, 4096, 8, True), (1024, 4160, 8, False),
    (2048, 16384, 8, True), (2048, 16448, 8, False), (1920, 8192, 8, False), (1024, 8192, 5, True), (1024, 8256, 5, False),
    (128, 4096, 4, True), (128, 4160, 4, False), (32768, 64, 8, True), (32896, 64, 1, False), (1056, 1024, 1, False)])
def test_kernel_by_shape_below(rows, cols, tokens, expected):
    linear = host.Nvfp4Sm100Linear.__new__(host.Nvfp4Sm100Linear)
    linear.rows, linear.cols = rows, cols
    need = host.gemv_tc_linear_scratch_bytes(cols)
    plan = lambda bytes_: SimpleNamespace(snapshot=lambda: SimpleNamespace(scratch_len_bytes=bytes_))
    assert linear._on_tensor_memory_below(plan(need), tokens) is expected
    assert linear._on_tensor_memory_below(plan(need - 256), tokens) is False
