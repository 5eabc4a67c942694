"""The fused cached token (``ops.decode_block``) against the operator-by-operator token, over the sizes where its tiles have
edges: batch rows around 16, 32 and 64, gate heads around 32 channels and one stage of the contraction."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _setup(batch, heads, head_width, dtype, mask, positions, seed=0):
    from griffin_b200 import RecurrentBlock, RecurrentBlockCache
    torch.manual_seed(seed)
    width = heads * head_width
    block = RecurrentBlock(48, width, gate_blocks=heads).to(DEV)
    with torch.no_grad():
        for bias in (block.rg_lru.recurrence_gate.bias, block.rg_lru.input_gate.bias, block.temporal_conv.bias):
            bias.normal_(std=0.3)
        block.temporal_conv.weight.normal_(std=0.5)
        block.rg_lru.Lambda[::5] = -2.0        # decays outside the polynomial's range
        for p in block.parameters():           # values that bf16 holds, so that both dtypes run on the same numbers
            p.copy_(p.to(torch.bfloat16).float())
    x = torch.randn(batch, 1, 48, device=DEV).to(torch.bfloat16)
    cache = RecurrentBlockCache(torch.randn(batch, width, device=DEV), torch.randn(batch, 3, width, device=DEV).to(torch.bfloat16),
                                torch.randint(-1, 5, (batch,), device=DEV))
    active = (torch.rand(batch, 1, device=DEV) < 0.7) if mask else None
    seg = torch.randint(0, 6, (batch, 1), device=DEV) if positions else None
    return block, x.to(dtype), RecurrentBlockCache(cache.rnn_state, cache.conv_state.to(dtype), cache.segment_position), active, seg


def _by_operators(block):
    block.rg_lru.recurrence_gate.register_forward_hook(lambda module, args, out: None)   # a hooked layer is called as it is
    return block


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("batch,heads,head_width,mask,positions", [
    (1, 2, 8, False, False), (3, 3, 24, True, False), (16, 2, 32, False, True), (17, 1, 40, True, True), (32, 2, 64, True, False),
    (33, 2, 72, False, False), (64, 1, 352, True, True), (65, 3, 48, True, False), (130, 2, 136, False, True)])
def test_fused_token_matches_the_operators(dtype, batch, heads, head_width, mask, positions, monkeypatch):
    from griffin_b200 import ops
    calls = []
    fused = ops.decode_block
    monkeypatch.setattr(ops, "decode_block", lambda *a: calls.append(1) or fused(*a))
    block, x, cache, active, seg = _setup(batch, heads, head_width, dtype, mask, positions)
    kept = [t.clone() for t in (cache.rnn_state, cache.conv_state, cache.segment_position)]
    with torch.no_grad():
        got, new = block.to(dtype)(x, cache, seg, active_mask=active, return_cache=True)
        assert calls == [1]
        # the yardstick runs in fp32 on the same values (they are bf16 numbers)
        ref_cache = type(cache)(cache.rnn_state, cache.conv_state.float(), cache.segment_position)
        want, ref = _by_operators(block.float())(x.float(), ref_cache, seg, active_mask=active, return_cache=True)
        assert calls == [1]
    for before, after in zip(kept, (cache.rnn_state, cache.conv_state, cache.segment_position)):
        assert torch.equal(before, after)
    # bf16: one rounding of x_in and of the conv output in front of the contraction, of y and of the output behind it;
    # the bound is the one the block's other bf16 tests use.  fp32: sums in another order.
    rel = 2e-2 if dtype == torch.bfloat16 else 1e-5
    for a, b in ((got, want), (new.rnn_state, ref.rnn_state), (new.conv_state, ref.conv_state)):
        a, b = a.double(), b.double()
        assert torch.isfinite(a).all()
        assert (a - b).norm() <= rel * b.norm().clamp_min(1e-30)
    assert torch.equal(new.segment_position, ref.segment_position)
    if mask:                                   # a padding row keeps its state and its position to the bit
        rows = ~active[:, 0]
        assert torch.equal(new.rnn_state[rows], cache.rnn_state[rows])
        assert torch.equal(new.conv_state[rows], cache.conv_state[rows])
        assert torch.equal(new.segment_position[rows], cache.segment_position[rows])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_batches_past_one_grid_axis(dtype):
    """262145 rows: one more than 65535 blocks of four rows hold.  Rows do not depend on each other, so the first and the
    last ones are what a call on them alone gives, to the bit."""
    from griffin_b200 import _lib, ops
    torch.manual_seed(0)
    batch, heads, bw = 262145, 1, 8
    D = heads * bw
    r = lambda *s: torch.randn(*s, device=DEV).to(dtype)
    shared = dict(conv_w=r(D, 4), conv_b=r(D), w_r=r(heads, bw, bw), b_r=r(heads, bw), w_i=r(heads, bw, bw), b_i=r(heads, bw),
                  lam=torch.randn(D, device=DEV))
    rows = dict(x_in=r(batch, D), branch=r(batch, D), conv_state=r(batch, 3, D), h=torch.randn(batch, D, device=DEV),
                position=torch.randint(0, 5, (batch,), device=DEV))
    whole = ops.decode_block(**rows, **shared)
    for part in (slice(0, 100), slice(batch - 97, batch)):
        alone = ops.decode_block(**{k: v[part] for k, v in rows.items()}, **shared)
        for a, b in zip(whole, alone):
            assert torch.equal(a[part], b)
    assert _lib.device_status() == 0


def test_very_large_batches_go_by_operators(monkeypatch):
    from griffin_b200 import ops
    block, x, cache, _, _ = _setup(65537, 1, 8, torch.bfloat16, False, False)
    monkeypatch.setattr(ops, "decode_block", None)
    with torch.no_grad():
        out, _ = block.bfloat16()(x, cache, return_cache=True)
    assert torch.isfinite(out).all()


class _Scale(torch.nn.Module):
    """A gate without any attribute of the layer it replaces."""

    def forward(self, x):
        return x * 0.5


def test_a_replaced_gate_goes_by_operators():
    block, x, cache, _, _ = _setup(3, 2, 16, torch.float32, False, False)
    block.rg_lru.group_gates = False
    block.rg_lru.recurrence_gate = _Scale()
    with torch.no_grad():
        out, new = block(x, cache, return_cache=True)
        # with gradients the token takes the scan kernels
        with torch.enable_grad():
            want, ref = block(x, cache, return_cache=True)
    torch.testing.assert_close(out, want, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(new.rnn_state, ref.rnn_state, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("cached", [False, True])
def test_gates_of_different_heads_run_as_modules(cached):
    """A gate of this package's own class with other heads than its partner's: neither fused form can read it."""
    from griffin_b200 import BlockDiagonalLinear
    block, x, cache, _, _ = _setup(3, 2, 24, torch.float32, False, False)
    gate = BlockDiagonalLinear(48, num_blocks=3).to(DEV)
    block.rg_lru.input_gate = gate
    with torch.no_grad():
        out, new = block(x, cache if cached else None, return_cache=True)
        block = _by_operators(block)
        want, ref = block(x, cache if cached else None, return_cache=True)
    torch.testing.assert_close(out, want, rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(new.rnn_state, ref.rnn_state, rtol=1e-5, atol=1e-6)
