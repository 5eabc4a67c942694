"""Arguments that the library would read or write out of range are refused on the host, before the library is reached: the
operators run here on CPU tensors with the CUDA requirement lifted and a library that fails the test when it is asked for."""

from __future__ import annotations

import pytest
import torch


class _Reached(Exception):
    pass


@pytest.fixture
def ops(monkeypatch):
    from griffin_b200 import _lib, ops

    def reached():
        raise _Reached
    monkeypatch.setattr(_lib, "load", reached)
    monkeypatch.setattr(ops, "_require_cuda", lambda *tensors: None)
    monkeypatch.setattr(ops, "_on", lambda t, name: ops._SAME_DEVICE)
    return ops


def _decode_args(dtype=torch.bfloat16, B=3, D=48, G=2):
    bw = D // G
    r = lambda *s: torch.randn(*s).to(dtype)
    return dict(x_in=r(B, D), branch=r(B, D), conv_w=torch.randn(D, 4), conv_b=r(D), conv_state=r(B, 3, D), w_r=r(G, bw, bw),
                b_r=r(G, bw), w_i=r(G, bw, bw), b_i=r(G, bw), lam=torch.randn(D), h=torch.randn(B, D),
                position=torch.zeros(B, dtype=torch.long), segment_pos=torch.zeros(B, dtype=torch.long),
                active=torch.ones(B, dtype=torch.bool))


def test_decode_block_takes_what_it_is_meant_for(ops):
    with pytest.raises(_Reached):
        ops.decode_block(**_decode_args())
    with pytest.raises(_Reached):
        ops.decode_block(**{**_decode_args(torch.float32), "branch": None, "conv_b": None, "segment_pos": None, "active": None})


@pytest.mark.parametrize("name,change", [
    ("h", lambda t: t.bfloat16()), ("h", lambda t: t[:2]), ("conv_state", lambda t: t[:, :2]), ("conv_state", lambda t: t.float()),
    ("position", lambda t: t.int()), ("position", lambda t: t[:2]), ("segment_pos", lambda t: t.int()),
    ("segment_pos", lambda t: t[:, None]), ("active", lambda t: t.long()), ("active", lambda t: t[:1]), ("branch", lambda t: t[:, :8]),
    ("branch", lambda t: t.float()), ("w_r", lambda t: t.float()), ("w_i", lambda t: t[:1]), ("w_r", lambda t: t[..., :8]),
    ("w_r", lambda t: t[:1]), ("b_r", lambda t: t.float()), ("b_i", lambda t: t[:1]), ("conv_w", lambda t: t[:, :3]),
    ("conv_w", lambda t: t.half()), ("conv_b", lambda t: t[:8]), ("lam", lambda t: t[:8]), ("lam", lambda t: t.double()),
    ("x_in", lambda t: t[0])])
def test_decode_block_refuses_other_shapes_and_dtypes(ops, name, change):
    args = _decode_args()
    args[name] = change(args[name])
    with pytest.raises((ValueError, TypeError)):
        ops.decode_block(**args)


def _plan_args(B=3, T=5):
    return dict(segment_pos=torch.zeros(B, T, dtype=torch.long), previous=torch.zeros(B, dtype=torch.long),
                active=torch.ones(B, T, dtype=torch.bool), reset=torch.zeros(B, T, dtype=torch.bool))


@pytest.mark.parametrize("name,change", [
    ("segment_pos", lambda t: t.int()), ("segment_pos", lambda t: t[:, :4]), ("previous", lambda t: t.int()),
    ("previous", lambda t: t[:1]), ("active", lambda t: t.long()), ("active", lambda t: t[:2]), ("reset", lambda t: t.float()),
    ("reset", lambda t: t[0]), ("active", lambda t: t.to("meta")), ("segment_pos", lambda t: t.to("meta"))])
def test_token_plan_refuses_other_shapes_dtypes_and_devices(ops, name, change):
    args = _plan_args()
    with pytest.raises(_Reached):
        ops.token_plan(3, 5, torch.device("cpu"), **args)
    args[name] = change(args[name])
    with pytest.raises((ValueError, RuntimeError)):
        ops.token_plan(3, 5, torch.device("cpu"), **args)


def test_token_plan_refuses_tensors_that_are_not_on_a_gpu():
    from griffin_b200 import ops
    with pytest.raises(RuntimeError):
        ops.token_plan(3, 5, torch.device("cpu"), **_plan_args())


def test_token_plan_makes_strided_masks_dense(ops, monkeypatch):
    seen = []
    ptr = ops._ptr
    monkeypatch.setattr(ops, "_ptr", lambda t: seen.append(t) or ptr(t))
    monkeypatch.setattr(ops, "_stream", lambda t: 0)
    monkeypatch.setattr(ops._lib, "load", lambda: type("L", (), {
        "rglru_token_plan_ws": staticmethod(lambda *a: 0), "rglru_token_plan_workspace_bytes": staticmethod(lambda *a: 0)}))
    args = _plan_args()
    args["active"] = torch.ones(5, 3, dtype=torch.bool).T
    args["segment_pos"] = torch.zeros(5, 3, dtype=torch.long).T
    ops.token_plan(3, 5, torch.device("cpu"), **args)
    assert len(seen) >= 6 and all(t is None or t.is_contiguous() for t in seen)


@pytest.mark.parametrize("one_call", [False, True])
@pytest.mark.parametrize("name,change", [
    ("h0", lambda t: t[:1]), ("h0", lambda t: t[:, :8]), ("h0", lambda t: t.to("meta")), ("tok", lambda t: t[:, :4]),
    ("tok", lambda t: t.int()), ("tok", lambda t: t.to("meta")), ("branch", lambda t: t.to("meta")),
    ("w_i", lambda t: t.to("meta")), ("lam", lambda t: t.to("meta"))])
def test_gated_layer_refuses_states_flags_and_branches_it_cannot_read(ops, monkeypatch, one_call, name, change):
    monkeypatch.setattr(ops, "_layer_in_library", lambda *a: one_call)
    monkeypatch.setattr(ops, "gated_supported", lambda *a: True)
    B, T, D, G = 2, 5, 128, 2
    w, b = torch.randn(G, D // G, D // G), torch.randn(G, D // G)
    args = dict(x=torch.randn(B, T, D), w_r=w, b_r=b, w_i=w, b_i=b, lam=torch.randn(D), h0=torch.randn(B, D),
                tok=torch.zeros(B, T, dtype=torch.uint8), branch=torch.randn(B, T, D))
    with torch.no_grad(), pytest.raises(_Reached):
        ops.rglru_gated(**args)
    args[name] = change(args[name])
    with torch.no_grad(), pytest.raises((ValueError, RuntimeError)):
        ops.rglru_gated(**args)


def test_a_cached_token_through_a_replaced_gate_is_not_taken_by_the_fused_form():
    """The decision reads nothing that a replaced layer need not have."""
    from griffin_b200 import RecurrentBlock

    class OnGpu:
        is_cuda, shape, dtype = True, (1, 1, 32), torch.float32
        element_size = staticmethod(lambda: 4)

    for replace in ("recurrence_gate", "input_gate"):
        block = RecurrentBlock(32, 64, gate_blocks=2)
        setattr(block.rg_lru, replace, torch.nn.Identity())
        with torch.no_grad():
            assert block._fused_token_parts(OnGpu(), None, None) is None
    block = RecurrentBlock(32, 64, gate_blocks=2)
    block.rg_lru = torch.nn.Identity()
    with torch.no_grad():
        assert block._fused_token_parts(OnGpu(), None, None) is None


@pytest.mark.parametrize("register", ["register_module_forward_hook", "register_module_forward_pre_hook",
                                      "register_module_full_backward_hook"])
def test_hooks_for_all_modules_keep_the_gates_modules(register):
    """A hook registered for every module has to see the gate projections, so they are called as the modules they are."""
    from griffin_b200 import RG_LRU, modules
    gate = RG_LRU(96, gate_blocks=2).recurrence_gate
    assert modules._is_stock(gate, modules.BlockDiagonalLinear)
    handle = getattr(torch.nn.modules.module, register)(lambda *args: None)
    try:
        assert not modules._is_stock(gate, modules.BlockDiagonalLinear)
    finally:
        handle.remove()
    assert modules._is_stock(gate, modules.BlockDiagonalLinear)
