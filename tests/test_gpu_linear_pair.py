"""``ops.linear_pair`` against two ``F.linear`` calls in float64: every gradient, with and without autocast, with one output
unused, and with an input that wants no gradient."""

from __future__ import annotations

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("mode", ["fp32", "bf16", "autocast", "autocast_bf16_input"])
@pytest.mark.parametrize("shape,n1,n2", [((1, 1, 8), 8, 16), ((2, 37, 24), 40, 8), ((3, 130, 768), 1024, 1000)])
@pytest.mark.parametrize("used", ["both", "first", "second", "no_dx"])
def test_linear_pair(mode, shape, n1, n2, used):
    from griffin_b200 import ops
    torch.manual_seed(0)
    width = shape[-1]
    params = torch.bfloat16 if mode == "bf16" else torch.float32
    inputs = torch.bfloat16 if mode in ("bf16", "autocast_bf16_input") else torch.float32
    out_dtype = torch.float32 if mode == "fp32" else torch.bfloat16
    make = lambda *s: torch.randn(*s, device=DEV).to(torch.bfloat16)      # values both types hold
    x = make(*shape).to(inputs).requires_grad_(used != "no_dx")
    ps = [t.to(params).requires_grad_(True) for t in (make(n1, width), make(n1), make(n2, width), make(n2))]
    d1, d2 = make(*shape[:2], n1).to(out_dtype), make(*shape[:2], n2).to(out_dtype)
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=mode.startswith("autocast")):
        y1, y2 = ops.linear_pair(x, *ps)
    assert y1.dtype == y2.dtype == out_dtype and type(y1.grad_fn).__name__ == "_LinearPairBackward"
    ref_x, ref_p = x.detach().double().requires_grad_(used != "no_dx"), [p.detach().double().requires_grad_(True) for p in ps]
    r1, r2 = F.linear(ref_x, ref_p[0], ref_p[1]), F.linear(ref_x, ref_p[2], ref_p[3])
    outs = {"first": ([y1], [r1], [d1]), "second": ([y2], [r2], [d2])}.get(used, ([y1, y2], [r1, r2], [d1, d2]))
    torch.autograd.backward(outs[0], outs[2])
    torch.autograd.backward(outs[1], [d.double() for d in outs[2]])
    # bf16 results: one rounding, two for the input gradient (2^-9 each); fp32 ones: fp32 sums of at most 1024 products.
    for a, b in zip([y1, y2, x.grad] + [p.grad for p in ps], [r1, r2, ref_x.grad] + [p.grad for p in ref_p]):
        assert (a is None) == (b is None)
        if a is None:
            continue
        bound = 1e-5 if a.dtype == torch.float32 else 2.0 ** -8
        assert a.shape == b.shape and (a.double() - b).norm() <= bound * b.norm()
    assert x.grad is None or x.grad.dtype == inputs
    assert all(p.grad is None or p.grad.dtype == params for p in ps)
