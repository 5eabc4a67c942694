"""Zeroing of padding rows in place against a select."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF, F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("rows,width,dtype", [(1, 8, BF), (7, 24, BF), (9, 4, F32), (1200, 768, BF), (33, 2560, F32)])
def test_zero_rows(rows, width, dtype):
    from griffin_b200 import _lib
    torch.manual_seed(rows)
    x = torch.randn(rows, width, device=DEV).to(dtype)
    keep = torch.rand(rows, device=DEV) < 0.5
    x[0, 0], keep[0] = float("nan"), False
    want = torch.where(keep[:, None], x, 0.0)
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.load().rglru_zero_rows(x.data_ptr(), keep.view(torch.uint8).data_ptr(), rows, width * x.element_size(), stream), "rows")
    assert torch.equal(x, want)
    assert _lib.load().rglru_zero_rows(x.data_ptr(), keep.data_ptr(), rows, 8, stream) != 0
