"""The block's small kernels: flag bytes and last positions from the masks against the tensor operations they stand for, and
the product with the GeLU branch against float64."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("batch,steps", [(1, 1), (3, 2), (2, 4), (5, 37), (2, 2047), (3, 2048), (2, 2049), (1, 5000), (40, 129)])
@pytest.mark.parametrize("given", ["active", "positions", "both", "cached", "cached_active", "cached_both", "full_mask"])
def test_token_plan_matches_the_tensor_operations(batch, steps, given):
    from griffin_b200 import modules, ops
    torch.manual_seed(steps)
    x = torch.empty(batch, steps, 1, device=DEV)
    active = seg = prev = None
    if given in ("active", "both", "cached_active", "cached_both"):
        length = torch.randint(0, steps + 1, (batch, 1), device=DEV)        # rows without any real token among them
        active = torch.arange(steps, device=DEV)[None] < length
    if given == "full_mask":
        active = torch.ones(batch, steps, dtype=torch.bool, device=DEV)
    if given in ("positions", "both", "cached_both"):
        seg = torch.randint(-2, 9, (batch, steps), device=DEV)
    if given.startswith("cached"):
        prev = torch.randint(-1, 6, (batch,), device=DEV)
    flags, last = ops.token_plan(batch, steps, DEV, segment_pos=seg, previous=prev, active=active)
    pos = modules._positions(x, seg, prev, active)
    with ops.library_ops():                                                  # the route of tensor operations
        want = modules.token_flags(batch, steps, DEV, reset=pos == 0, active=active, segment_pos=pos,
                                   padded=None if active is None else ~active.all())
    assert torch.equal(flags, want)
    assert torch.equal(last, modules._last_real_position(pos, active, prev))


@pytest.mark.parametrize("batch,steps", [(1, 1), (3, 37), (2, 2050)])
@pytest.mark.parametrize("given", ["reset", "active", "both"])
def test_layer_flags_match_the_tensor_operations(batch, steps, given):
    from griffin_b200 import modules, ops
    torch.manual_seed(0)
    reset = (torch.rand(batch, steps, device=DEV) < 0.3) if given != "active" else None
    active = (torch.rand(steps, batch, device=DEV) < 0.6).T if given != "reset" else None     # not contiguous
    got = modules.token_flags(batch, steps, torch.device(DEV, torch.cuda.current_device()), reset=reset, active=active)
    with ops.library_ops():
        want = modules.token_flags(batch, steps, DEV, reset=reset, active=active)
    assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 5), (1, 7, 8), (3, 129, 72), (2, 255, 1000)])
def test_gelu_mul(shape, dtype):
    from griffin_b200 import ops
    torch.manual_seed(0)
    y, g, d = (torch.randn(*shape, device=DEV).mul_(s).to(dtype) for s in (1.0, 3.0, 1.0))
    g.view(-1)[:1] = -40.0
    ly, lg = y.clone().requires_grad_(True), g.clone().requires_grad_(True)
    out = ops.gelu_mul(ly, lg)
    out.backward(d)
    ry, rg = y.double().requires_grad_(True), g.double().requires_grad_(True)
    ref = ry * torch.nn.functional.gelu(rg, approximate="tanh")
    ref.backward(d.double())
    # One rounding to the type, 2^-9 at most relative to each value for bf16; fp32: a handful of roundings and two
    # hardware functions good to 2^-22.
    bound = 2.0 ** -9 if dtype == torch.bfloat16 else 2e-6
    for a, b in ((out, ref), (ly.grad, ry.grad), (lg.grad, rg.grad)):
        assert a.dtype == dtype and a.shape == b.shape
        assert (a.double() - b).norm() <= bound * b.norm().clamp_min(1e-30)


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 1e30, -1e30])
def test_gelu_mul_far_out(value):
    from griffin_b200 import ops
    y, g = torch.full((8,), 2.0, device=DEV), torch.full((8,), value, device=DEV)
    want = y * torch.nn.functional.gelu(g, approximate="tanh")
    torch.testing.assert_close(ops.gelu_mul(y, g), want, equal_nan=True)


@pytest.mark.parametrize("batch,steps", [(1, 70000), (2, 32769), (9, 8192), (1024, 2048), (70000, 1)])
@pytest.mark.parametrize("hole", [None, 0, 0.5, 1])
def test_token_plan_of_large_masks(batch, steps, hole):
    """Padding is looked for in parts: none, or one token of it at the first, a middle and the last place."""
    from griffin_b200 import modules, ops
    x = torch.empty(batch, steps, 1, device=DEV)
    storage = torch.ones(batch * steps + 3, dtype=torch.bool, device=DEV)
    for shift in (0, 3):                                  # a mask that does not start on a 16-byte boundary either
        active = storage[shift:shift + batch * steps].view(batch, steps)
        active.fill_(True)
        if hole is not None:
            active.view(-1)[int(hole * (batch * steps - 1))] = False
        flags, last = ops.token_plan(batch, steps, DEV, active=active)
        pos = modules._positions(x, None, None, active)
        with ops.library_ops():
            want = modules.token_flags(batch, steps, DEV, reset=pos == 0, active=active, segment_pos=pos, padded=~active.all())
        assert torch.equal(flags, want)
        assert torch.equal(last, modules._last_real_position(pos, active, None))
