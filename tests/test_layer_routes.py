"""Which projections a layer takes, decided on the host from sizes and the caller's settings (no device needed)."""

from __future__ import annotations

import pytest
import torch


@pytest.fixture
def ops(monkeypatch):
    from griffin_b200 import ops
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(ops, "_gemms_capturable", lambda *a: True)
    return ops


@pytest.fixture
def precision():
    before = torch.get_float32_matmul_precision()
    yield torch.set_float32_matmul_precision
    torch.set_float32_matmul_precision(before)


def _x(rows, width, dtype):
    return torch.empty(1, rows, width, device="meta", dtype=dtype)


def test_the_callers_tf32_setting_is_seen(ops, precision):
    for setting, allowed in (("highest", False), ("high", True), ("medium", True)):
        precision(setting)
        assert ops._tf32_allowed() is allowed


@pytest.mark.parametrize("dtype,rows,width,bw,grad,eager,captured", [
    (torch.bfloat16, 16384, 1024, 64, True, True, False), (torch.bfloat16, 16385, 1024, 64, True, False, False),
    (torch.bfloat16, 16384, 1024, 64, False, False, False), (torch.bfloat16, 8192, 1024, 64, False, True, False),
    (torch.bfloat16, 16384, 64, 16, True, True, True), (torch.bfloat16, 16384, 64, 16, False, True, False),
    (torch.float32, 8192, 512, 128, True, True, False), (torch.float32, 8192, 512, 32, True, True, True),
    (torch.float32, 65536, 256, 16, False, True, True), (torch.float32, 4096, 2048, 128, True, False, False),
    (torch.bfloat16, 2, 8 * 65536, 8, True, False, False)])
def test_projections_by_size(ops, monkeypatch, dtype, rows, width, bw, grad, eager, captured):
    assert ops._layer_in_library(_x(rows, width, dtype), bw, grad) is eager
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert ops._layer_in_library(_x(rows, width, dtype), bw, grad) is captured


def test_projections_where_tf32_is_allowed(ops, precision, monkeypatch):
    x = _x(8192, 512, torch.float32)
    assert ops._layer_in_library(x, 32, False) and ops._layer_in_library(x, 128, True)
    precision("high")
    assert not ops._layer_in_library(x, 128, False) and ops._layer_in_library(x, 128, True)
    assert ops._layer_in_library(_x(8192, 512, torch.bfloat16), 128, False)          # no business of bf16's
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert not ops._layer_in_library(x, 32, True) and not ops._layer_in_library(x, 32, False)
    assert ops._layer_in_library(_x(65536, 256, torch.float32), 16, True)


def test_what_was_not_warmed_up_is_captured_without_gemms(ops, monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    monkeypatch.setattr(ops, "_gemms_capturable", lambda *a: False)
    assert ops._layer_in_library(_x(16384, 1024, torch.bfloat16), 64, True)
    assert not ops._layer_in_library(_x(16385, 1024, torch.bfloat16), 64, True)
