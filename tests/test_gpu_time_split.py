"""Calls with too few (batch row, channel tile) pairs to fill the machine are split along time over the blocks of a
cluster.  Lengths around the places where a block of the cluster runs out of chunks, against the fp64 oracle and against
the raw scan's fp64 recurrence."""

from __future__ import annotations

import pytest
import torch

from oracle import rglru_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"

# one chunk; just over one; a whole round of eight; a round and one step (seven blocks idle in the last); odd rounds
LENGTHS = [64, 65, 512, 513, 64 * 17 - 1, 64 * 21]


@pytest.mark.parametrize("steps", LENGTHS)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("masked", [False, True])
def test_split_scan_against_oracle(steps, dtype, masked):
    from griffin_b200 import _lib, ops
    from griffin_b200.modules import token_flags
    B, D = 2, 200                                     # four tiles a row, the last one cut
    gen = torch.Generator().manual_seed(steps)
    x, u_r, u_i, dy = (torch.randn(B, steps, D, generator=gen).to(dtype) for _ in range(4))
    lam = orc.init_lambda(D, 8.0, gen)
    h0, dh = torch.randn(B, D, generator=gen), torch.randn(B, D, generator=gen)
    reset = active = None
    if masked:
        reset = torch.rand(B, steps, generator=gen) < 0.02
        active = torch.ones(B, steps, dtype=torch.bool)
        active[-1, steps - steps // 3:] = False
    leaves = [t.to(DEV).requires_grad_(True) for t in (x, u_r, u_i, lam, h0)]
    flags = None if not masked else token_flags(B, steps, DEV, reset=reset.to(DEV), active=active.to(DEV))
    y, h_last = ops.rglru(*leaves, flags)
    ((y.float() * dy.to(DEV).float()).sum() + (h_last * dh.to(DEV)).sum()).backward()
    want = orc.rglru_backward_linear(x.double(), u_r.double(), u_i.double(), lam.double(), dy.double(), h0=h0, dh_last=dh,
                                     reset=reset, active=active)
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    got = dict(y=y, h_last=h_last, dx=leaves[0].grad, du_r=leaves[1].grad, du_i=leaves[2].grad, dLambda=leaves[3].grad,
               dh0=leaves[4].grad)
    for key, value in got.items():
        assert orc.rel_l2(value, want[key]) <= tol, key
    assert _lib.device_status() == 0


@pytest.mark.parametrize("merge", [False, True])
@pytest.mark.parametrize("steps", [65, 64 * 9 + 3])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_split_layer_against_oracle(steps, dtype, merge):
    from griffin_b200 import _lib, ops
    B, D, G = 1, 128, 2
    bw = D // G
    gen = torch.Generator().manual_seed(steps + merge)
    rnd = lambda *s: torch.randn(*s, generator=gen)
    x, branch, dout = rnd(B, steps, D).to(dtype), rnd(B, steps, D).to(dtype), rnd(B, steps, D).to(dtype)
    w = [(rnd(G, bw, bw) / bw ** 0.5).to(dtype).float(), rnd(G, bw) * 0.3, (rnd(G, bw, bw) / bw ** 0.5).to(dtype).float(),
         rnd(G, bw) * 0.3]
    lam = orc.init_lambda(D, 8.0, gen)
    names = ("recurrence_gate.weight", "recurrence_gate.bias", "input_gate.weight", "input_gate.bias")
    ref = {k: v.double().requires_grad_(True) for k, v in zip(names + ("Lambda",), w + [lam])}
    xd, bd = x.double().requires_grad_(True), branch.double().requires_grad_(True)
    y, _ = orc.rglru_layer_linear_backward(xd, ref)
    out_ref = y * torch.nn.functional.gelu(bd, approximate="tanh") if merge else y
    (out_ref * dout.double()).sum().backward()
    dev = [t.to(DEV).requires_grad_(True) for t in w + [lam]]
    xg, bg = x.to(DEV).requires_grad_(True), branch.to(DEV).requires_grad_(True)
    out, _ = ops.rglru_grouped(xg, *dev[:4], dev[4], branch=bg if merge else None)
    (out.float() * dout.to(DEV).float()).sum().backward()
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    pairs = [("out", out, out_ref), ("dx", xg.grad, xd.grad)] + [(k, g.grad, ref[k].grad) for k, g in zip(names + ("Lambda",), dev)]
    if merge:
        pairs.append(("dbranch", bg.grad, bd.grad))
    for key, got, want in pairs:
        assert orc.rel_l2(got, want) <= tol, key
    assert _lib.device_status() == 0


@pytest.mark.parametrize("steps", LENGTHS)
@pytest.mark.parametrize("width", [32, 100])
def test_split_raw_scan(steps, width):
    from griffin_b200 import _lib, ops
    gen = torch.Generator().manual_seed(steps + width)
    a = torch.rand(2, steps, width, generator=gen) * 0.3 + 0.7
    b, dy = torch.randn(2, steps, width, generator=gen), torch.randn(2, steps, width, generator=gen)
    h0 = torch.randn(2, width, generator=gen)
    ref = [t.double().requires_grad_(True) for t in (a, b, h0)]
    want = orc.linear_scan(*ref)
    (want * dy.double()).sum().backward()
    dev = [t.to(DEV).requires_grad_(True) for t in (a, b, h0)]
    got = ops.linear_scan(*dev)
    (got * dy.to(DEV)).sum().backward()
    assert orc.rel_l2(got, want) <= 1e-5
    for g, r in zip(dev, ref):
        assert orc.rel_l2(g.grad, r.grad) <= 1e-5
    assert _lib.device_status() == 0
