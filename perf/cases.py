"""The work whose speed this package is judged by, as a user's program has it done through the public entry points.

Six kinds of call, each over the sizes it is used at:

* ``scan``    training step of the bare operator ``ops.rglru`` on gate pre-activations that are already there;
* ``affine``  training step of the bare fp32 operator ``ops.linear_scan``;
* ``layer``   training step of the ``RG_LRU`` module (gate projections and recurrence);
* ``block``   training step of the ``RecurrentBlock`` module (projections, conv, recurrence, branch product);
* ``prefill`` ``RecurrentBlock`` over a prompt without gradients, returning the cache for decoding;
* ``decode``  one token of ``RecurrentBlock`` from a cache.

A training step is a forward and a backward from a given output gradient; it returns the outputs and every gradient.
"""

import contextlib

import torch

from griffin_b200 import RG_LRU, RecurrentBlock, RecurrentBlockCache, ops

_DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
_BYTES = {"bf16": 2, "fp32": 4}


def listed():
    return [
        # the benchmark's headline: the recurrence alone at the ordinary training shape, bf16 tensors
        dict(name="scan_bf16", kind="scan", dtype="bf16", batch=8, steps=2048, width=1024, masks="none"),
        # the operator a kernel user calls with decays of his own, on odd sizes (last rows and columns of every tile cut off)
        dict(name="affine_fp32_ragged", kind="affine", dtype="fp32", batch=3, steps=1999, width=1000),
        # the smallest layer call of the configurations, fp32: launches and host time
        dict(name="layer_fp32_small", kind="layer", dtype="fp32", batch=2, steps=256, width=256, heads=4, masks="none"),
        # full precision training with document resets and padding, odd batch and length, gate heads of 48 channels
        dict(name="layer_fp32_masked", kind="layer", dtype="fp32", batch=5, steps=1537, width=768, heads=16, masks="both"),
        # the ordinary layer of the 100M model's width
        dict(name="layer_bf16", kind="layer", dtype="bf16", batch=8, steps=2048, width=1024, heads=16, masks="none"),
        # one long document per GPU: nothing to share among the batch
        dict(name="layer_bf16_long", kind="layer", dtype="bf16", batch=1, steps=16384, width=1024, heads=16, masks="none"),
        # the wide, long layer of the largest configuration, one GPU's eighth of its batch
        dict(name="layer_bf16_wide", kind="layer", dtype="bf16", batch=8, steps=8192, width=5632, heads=16, masks="none"),
        # the whole temporal-mixing block in bf16 at the benchmark's shape, branch product folded into the scan
        dict(name="block_bf16", kind="block", dtype="bf16", autocast=False, fold_merge=True, packed=False, batch=16,
             steps=2048, input=768, width=1024, heads=16),
        # the block as the language model's training loop runs it: fp32 parameters under bf16 autocast, packed documents
        dict(name="block_autocast_packed", kind="block", dtype="fp32", autocast=True, fold_merge=False, packed=True, batch=8,
             steps=2048, input=768, width=1024, heads=16),
        # prompts of different lengths in one batch, padded on the right
        dict(name="prefill_padded", kind="prefill", dtype="bf16", padding="right", batch=6, steps=1200, input=768, width=1024,
             heads=16),
        # one user's next token
        dict(name="decode_single", kind="decode", dtype="bf16", batch=1, input=768, width=1024, heads=16),
        # the next token of a full serving batch at the largest configuration's width
        dict(name="decode_batch", kind="decode", dtype="bf16", batch=512, input=4096, width=5632, heads=16),
    ]


def _between(rng, low, high):
    """A whole number whose logarithm is spread evenly over [low, high]."""
    return max(low, min(high, round(low * (high / low) ** rng.random())))


def draw(rng):
    kind = rng.choice(["scan", "affine", "layer", "layer", "block", "prefill", "decode", "decode"])
    heads = rng.choice([4, 8, 16, 16])
    width = heads * 8 * _between(rng, max(1, 256 // (8 * heads)), 5632 // (8 * heads))   # heads of a multiple of 8 channels
    if kind in ("scan", "affine"):
        if rng.random() < 0.2:
            width += rng.randint(1, 7)           # a width no vector load divides
        batch = _between(rng, 1, 32)
        steps = _between(rng, 64, max(64, min(16384, 67108864 // (batch * width))))
        if kind == "affine":
            return dict(kind=kind, dtype="fp32", batch=batch, steps=steps, width=width)
        return dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "fp32"]), batch=batch, steps=steps, width=width,
                    masks=rng.choice(["none", "none", "resets", "padding", "both"]))
    if kind == "layer":
        batch = _between(rng, 1, 32)
        steps = _between(rng, 64, max(64, min(16384, 67108864 // (batch * width))))
        return dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "fp32"]), batch=batch, steps=steps, width=width, heads=heads,
                    masks=rng.choice(["none", "none", "resets", "padding", "both"]))
    input_dim = 8 * _between(rng, 16, 512)
    if kind == "decode":
        return dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "fp32"]), batch=_between(rng, 1, 512), input=input_dim,
                    width=width, heads=heads)
    if kind == "prefill":
        batch = _between(rng, 1, 32)
        steps = _between(rng, 16, max(16, min(8192, 33554432 // (batch * width))))
        return dict(kind=kind, dtype="bf16", padding=rng.choice(["none", "right", "right", "left"]), batch=batch, steps=steps,
                    input=input_dim, width=width, heads=heads)
    batch = _between(rng, 1, 32)
    steps = _between(rng, 64, max(64, min(8192, 33554432 // (batch * width))))
    autocast = rng.random() < 0.5
    return dict(kind=kind, dtype="fp32" if autocast else "bf16", autocast=autocast, fold_merge=rng.random() < 0.5,
                packed=rng.random() < 0.5, batch=batch, steps=steps, input=input_dim, width=width, heads=heads)


def _normal(gen, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(dtype)


def _lengths(gen, batch, steps):
    """Real tokens per row: between half and all of the row, one row full."""
    n = torch.randint(max(1, steps // 2), steps + 1, (batch,), device="cuda", generator=gen)
    n[0] = steps
    return n


def _documents(gen, batch, steps):
    """Positions inside the documents packed into every row (about four each)."""
    start = torch.rand(batch, steps, device="cuda", generator=gen) < 4.0 / steps
    start[:, 0] = True
    at = torch.arange(steps, device="cuda").expand(batch, steps)
    return at - torch.where(start, at, torch.zeros_like(at)).cummax(dim=1).values


def _gate_biases(gen, layer):
    """A trained layer's gate biases are not the zeros of its initialisation."""
    with torch.no_grad():
        for gate in (layer.recurrence_gate, layer.input_gate):
            gate.bias.copy_(_normal(gen, *gate.bias.shape, scale=0.3))


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dtype = case["kind"], _DTYPES[case["dtype"]]
    batch, width = case["batch"], case["width"]
    state = {"kind": kind}

    if kind in ("scan", "layer"):
        steps = case["steps"]
        shape = (batch, steps, width)
        resets = _documents(gen, batch, steps) == 0 if case["masks"] in ("resets", "both") else None
        active = None
        if case["masks"] in ("padding", "both"):
            active = torch.arange(steps, device="cuda")[None, :] < _lengths(gen, batch, steps)[:, None]
        state["x"] = _normal(gen, *shape, dtype=dtype).requires_grad_(True)
        state["dy"] = _normal(gen, *shape, dtype=dtype)
        if kind == "layer":
            with torch.device("cuda"):
                layer = RG_LRU(width, gate_blocks=case["heads"])
            _gate_biases(gen, layer)
            state.update(layer=layer.to(dtype), resets=resets, active=active)
        else:
            from griffin_b200 import token_flags
            state["u_r"] = _normal(gen, *shape, dtype=dtype).requires_grad_(True)
            state["u_i"] = _normal(gen, *shape, dtype=dtype).requires_grad_(True)
            decay = torch.rand(width, device="cuda", generator=gen) * 0.099 + 0.9
            state["lam"] = torch.logit(decay.pow(1.0 / 8.0)).requires_grad_(True)
            state["flags"] = token_flags(batch, steps, torch.device("cuda"), reset=resets, active=active)
        return state

    if kind == "affine":
        shape = (batch, case["steps"], width)
        state["decay"] = (torch.rand(*shape, device="cuda", generator=gen) * 0.3 + 0.7).requires_grad_(True)
        state["drive"] = _normal(gen, *shape).requires_grad_(True)
        state["h0"] = _normal(gen, batch, width).requires_grad_(True)
        state["dy"] = _normal(gen, *shape)
        return state

    with torch.device("cuda"):
        block = RecurrentBlock(case["input"], width, gate_blocks=case["heads"], fold_merge=case.get("fold_merge", False))
    _gate_biases(gen, block.rg_lru)
    state["block"] = block = block.to(dtype)
    if kind == "block":
        steps = case["steps"]
        out_dtype = torch.bfloat16 if case["autocast"] else dtype
        state["x"] = _normal(gen, batch, steps, case["input"], dtype=dtype).requires_grad_(True)
        state["dy"] = _normal(gen, batch, steps, case["input"], dtype=out_dtype)
        state["positions"] = _documents(gen, batch, steps) if case["packed"] else None
        state["autocast"] = case["autocast"]
    elif kind == "prefill":
        steps = case["steps"]
        state["x"] = _normal(gen, batch, steps, case["input"], dtype=dtype)
        at, n = torch.arange(steps, device="cuda")[None, :], _lengths(gen, batch, steps)[:, None]
        state["active"] = {"none": None, "right": at < n, "left": at >= steps - n}[case["padding"]]
    else:
        state["x"] = _normal(gen, batch, 1, case["input"], dtype=dtype)
        state["cache"] = RecurrentBlockCache(_normal(gen, batch, width), _normal(gen, batch, 3, width, dtype=dtype),
                                             torch.randint(3, 4096, (batch,), device="cuda", generator=gen))
    return state


def _cache_parts(cache):
    return [cache.rnn_state, cache.conv_state, cache.segment_position]


def run(state):
    kind, x = state["kind"], state.get("x")
    if kind == "scan":
        leaves = [x, state["u_r"], state["u_i"], state["lam"]]
        for t in leaves:
            t.grad = None
        y, h_last = ops.rglru(x, state["u_r"], state["u_i"], state["lam"], None, state["flags"])
        y.backward(state["dy"])
        return [y.detach(), h_last.detach()] + [t.grad for t in leaves]
    if kind == "affine":
        leaves = [state["decay"], state["drive"], state["h0"]]
        for t in leaves:
            t.grad = None
        y = ops.linear_scan(*leaves)
        y.backward(state["dy"])
        return [y.detach()] + [t.grad for t in leaves]
    if kind == "layer":
        layer = state["layer"]
        layer.zero_grad(set_to_none=True)
        x.grad = None
        y, h_last = layer(x, reset_mask=state["resets"], active_mask=state["active"], return_state=True)
        y.backward(state["dy"])
        return [y.detach(), h_last.detach(), x.grad] + [p.grad for p in layer.parameters()]
    block = state["block"]
    if kind == "block":
        block.zero_grad(set_to_none=True)
        x.grad = None
        with torch.autocast("cuda", dtype=torch.bfloat16) if state["autocast"] else contextlib.nullcontext():
            y = block(x, None, state["positions"])
        y.backward(state["dy"])
        return [y.detach(), x.grad] + [p.grad for p in block.parameters()]
    with torch.no_grad():
        if kind == "prefill":
            y, cache = block(x, active_mask=state["active"], return_cache=True)
        else:
            y, cache = block(x, state["cache"], return_cache=True)
    return [y] + _cache_parts(cache)


def work(case):
    """Bytes: every tensor a pass is given or returns, once per direction that needs it (a backward reads its forward's
    inputs again; nothing in between is counted).  Flops: the projections; the recurrence's own are not worth counting."""
    size, batch, width = _BYTES[case["dtype"]], case["batch"], case["width"]
    tokens = batch * case.get("steps", 1)
    n = tokens * width
    kind = case["kind"]
    if kind == "scan":       # forward x, u_r, u_i -> y; backward dy, x, u_r, u_i -> dx, du_r, du_i
        return {"bytes": 11 * n * size, "flops": 0}
    if kind == "affine":     # forward decay, drive -> h; backward dh, decay, h -> d decay, d drive
        return {"bytes": 8 * n * size, "flops": 0}
    gate = 2 * width * width // case["heads"]
    if kind == "layer":      # forward x -> y; backward dy, x -> dx; the gate weights and their gradients
        return {"bytes": 5 * n * size + 3 * gate * size, "flops": 3 * 2 * tokens * gate}
    weights = 3 * case["input"] * width + gate
    m = tokens * case["input"]
    if kind == "block":      # forward x -> y; backward dy, x -> dx; the weights and their gradients
        return {"bytes": 5 * m * size + 3 * weights * size, "flops": 3 * 2 * tokens * weights}
    states = 2 * batch * width * (4 + 3 * size)
    if kind == "prefill":
        return {"bytes": 2 * m * size + weights * size + states // 2, "flops": 2 * tokens * weights}
    return {"bytes": 2 * m * size + weights * size + states, "flops": 2 * tokens * weights}


def tolerance(case):
    # bf16 against the same path on fp32 tensors of the same values: up to 2.6e-3 for the layer and the recurrence, 4.5e-3
    # for a token of the block, 6e-3 for the gradients of the block.  fp32 against the sequential scan: 2e-7 to 1e-6.
    if case["kind"] == "block":
        return {"rel": 2e-2}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 1e-5}
