"""Parameters and buffers that begin anywhere their element type allows (views into one flat buffer of parameters, say)."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _off_boundary(t):
    """A copy of ``t`` four bytes past a 16-byte boundary."""
    shift = 4 // t.element_size()
    return torch.empty(t.numel() + shift, device=t.device, dtype=t.dtype)[shift:].view(t.shape).copy_(t)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("batch,width", [(1, 64), (3, 200), (80, 64)])      # (80 rows: more than one round of the fold)
def test_lambda_off_a_16_byte_boundary(batch, width, dtype):
    """The backward's fold of dLambda reads Lambda four at a time only where it may: same bits either way."""
    from griffin_b200 import _lib, ops
    torch.manual_seed(0)
    x, u_r, u_i, dy = (torch.randn(batch, 70, width, device=DEV).to(dtype) for _ in range(4))
    lam = torch.randn(width, device=DEV) + 4

    def grads(value):
        leaves = [t.clone().requires_grad_(True) for t in (x, u_r, u_i)]
        value = value.detach().requires_grad_(True)
        y, _ = ops.rglru(*leaves, value)
        y.backward(dy)
        return [y.detach(), value.grad] + [t.grad for t in leaves]
    shifted = _off_boundary(lam)
    assert shifted.data_ptr() % 16 == 4
    for a, b in zip(grads(lam), grads(shifted)):
        assert torch.equal(a, b)
    assert _lib.device_status() == 0


def test_lambda_gradient_and_workspace_off_a_16_byte_boundary():
    """The C entry points ask for four-byte alignment of Lambda, its gradient and the workspace."""
    from griffin_b200 import _lib, ops
    torch.manual_seed(0)
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    B, T, D = 2, 70, 128
    x, u_r, u_i, dy = (torch.randn(B, T, D, device=DEV) for _ in range(4))
    lam = torch.randn(D, device=DEV) + 4
    got = []
    for move in (lambda t: t, _off_boundary):
        lam2, dlam = move(lam), move(torch.zeros(D, device=DEV))
        ws = move(torch.zeros(ops.workspace_bytes(B, T, D) // 4, device=DEV))
        y, dx, dr, di = (torch.empty_like(x) for _ in range(4))
        nbytes = ws.numel() * 4
        p = lambda t: t.data_ptr()
        _lib.check(lib.rglru_fwd(p(x), p(u_r), p(u_i), p(lam2), None, None, p(y), None, p(ws), nbytes, B, T, D, 8.0, _lib.F32, st), "fwd")
        _lib.check(lib.rglru_bwd(p(dy), None, p(x), p(u_r), p(u_i), p(lam2), None, None, p(ws), nbytes, p(dx), p(dr), p(di), p(dlam),
                                 None, B, T, D, 8.0, _lib.F32, st), "bwd")
        got.append([y, dx, dr, di, dlam.clone()])
    for a, b in zip(*got):
        assert torch.equal(a, b)
    assert _lib.device_status() == 0
