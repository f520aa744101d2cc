"""Which matrices the fp8 quantiser kernel takes: those that its launch can index; the PyTorch forms serve the others."""
from types import SimpleNamespace

import pytest
import torch


@pytest.mark.parametrize("rows,cols,ok", [(1, 128, True), (65535 * 128, 128, True), (65535 * 128 + 1, 128, False), (2 ** 23 - 1, 128, False),
                                          (0, 128, False), (4, 0, False), (4, 130, False)])
def test_row_and_column_limits(monkeypatch, rows, cols, ok):
    from mindspeed_b200.ops import gemm_fp8 as F
    monkeypatch.setattr(F.loader, "lib", lambda: object())
    x = SimpleNamespace(is_cuda=True, dtype=torch.bfloat16, shape=(rows, cols), is_contiguous=lambda: True, data_ptr=lambda: 256)
    assert bool(F._quant_ok(x, torch.float8_e4m3fn)) is ok
