"""Which of the two small-token kernels `Nvfp4Sm100Linear` takes: a rule on rows, columns, token rows and the plan's scratch."""
from types import SimpleNamespace

import pytest

from augur_v100_b200 import host


@pytest.mark.parametrize("rows,cols,tokens,expected", [
    (17408, 5120, 1, True), (17408, 5120, 8, True), (4096, 8192, 8, True), (4096, 8064, 8, False),      # 2^25 weights, and one block column less
    (3968, 8704, 5, False), (3968, 8704, 4, True), (2560, 13184, 4, True), (2432, 13824, 1, False),     # few rows: by the token rows
    (1024, 32768, 1, False), (17440, 5120, 8, False), (1 << 18, 128, 8, True), ((1 << 18) + 128, 128, 8, False)])
def test_kernel_by_shape(rows, cols, tokens, expected):
    linear = host.Nvfp4Sm100Linear.__new__(host.Nvfp4Sm100Linear)
    linear.rows, linear.cols = rows, cols
    need = host.gemv_tc_linear_scratch_bytes(cols)
    plan = lambda bytes_: SimpleNamespace(snapshot=lambda: SimpleNamespace(scratch_len_bytes=bytes_))
    assert linear._on_tensor_memory(plan(need), tokens) is expected
    assert linear._on_tensor_memory(plan(need - 256), tokens) is False


# What `bind` makes of it, below the line of the large weights too: those keep the kernel that multiplies every activation as it is.
@pytest.mark.parametrize("rows,cols,tokens,expected", [
    (17408, 5120, 8, "tensor memory"), (2560, 13184, 4, "tensor memory"), (2560, 13184, 8, "exact"), (3072, 12288, 8, "exact"), (2048, 16384, 8, "exact"),
    (3968, 8704, 5, "exact"), (4096, 8064, 1, "exact"), (4096, 4096, 4, "exact"), (2048, 5120, 8, "exact"), (1024, 5120, 1, "exact"), (1024, 4096, 8, "exact"),
    (128, 64, 1, "exact"), (32768, 64, 8, "exact"), (17440, 5120, 8, "exact")])
def test_bind_by_shape(monkeypatch, rows, cols, tokens, expected):
    monkeypatch.setattr(host.Nvfp4Sm100TcProjection, "bind", classmethod(lambda cls, plan, weight, x, out=None: ("tensor memory", weight)))
    monkeypatch.setattr(host.Nvfp4Sm100Projection, "bind", classmethod(lambda cls, plan, weight, x, out=None: ("exact", weight)))
    linear = host.Nvfp4Sm100Linear.__new__(host.Nvfp4Sm100Linear)
    linear.rows, linear.cols, linear.small, linear.wide = rows, cols, "small", "wide"
    plan = SimpleNamespace(snapshot=lambda: SimpleNamespace(scratch_len_bytes=1 << 30))
    bound = linear.bind(plan, SimpleNamespace(shape=(tokens, cols)))
    assert bound == (expected, "wide" if expected == "tensor memory" else "small")
