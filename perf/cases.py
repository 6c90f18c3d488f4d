"""What a user of this package runs, as measurable cases.

A case is a dict of plain values.  ``kind`` names the entry point:

* ``stack``      - ``PairformerModule``: the pair track and the single track of a trunk.
* ``pair_stack`` - ``PairformerNoSeqModule``: the pair track alone (template and MSA stacks).
* ``attention``  - ``TriangleAttentionStartingNode`` then ``TriangleAttentionEndingNode``, with ``transition`` also the
  SwiGLU ``Transition``: the layers swapped into a trunk of somebody else's.
* ``trimul``     - ``TriangleMultiplicationNode`` outgoing, then incoming.
* ``transition`` - ``Transition`` (``relu`` false) or ``PairTransition`` (``relu`` true) with a pair mask.

Every path is a forward pass in bfloat16 (the package is an inference runtime).  ``tokens`` is the padded extent, and
the valid tokens of the batch items lie evenly between ``valid`` and ``tokens``, ``valid`` first.
"""

import math

import torch

import bionemo_inference_runtime_b200 as b200

C_Z, C_S, HEADS_S = 128, 384, 16


def _stack(name, kind, tokens, valid, *, blocks, graph, batch=1, f32=False):
    return {"name": name, "kind": kind, "tokens": tokens, "valid": valid, "batch": batch, "blocks": blocks, "graph": graph,
            "f32": f32}


def _attention(name, tokens, valid, *, batch=1, transition=False, holes=False):
    return {"name": name, "kind": "attention", "tokens": tokens, "valid": valid, "batch": batch, "transition": transition,
            "holes": holes}


def listed():
    return [
        # A peptide through the two attention layers: nothing but launches and host work.
        _attention("attention_48", 48, 48),
        # A template stack over a small chain, replayed from a CUDA graph.
        _stack("pair_stack_graph_80", "pair_stack", 80, 80, blocks=4, graph=True),
        # The default trunk (8 blocks, fp32 triangle-multiplication outputs) on a small protein of an odd length in a
        # bucket of 120 tokens, without a graph: every request has another length.
        _stack("stack_120", "stack", 120, 113, blocks=8, graph=False, f32=True),
        # A served bucket of a common size, replayed from a CUDA graph.
        _stack("stack_graph_256", "stack", 256, 256, blocks=8, graph=True),
        # A few ragged proteins in one batch.
        _stack("stack_4x200", "stack", 200, 131, blocks=2, graph=False, batch=4),
        # Four blocks of the 48-block trunk at 768 tokens, the size large complexes are cropped to.
        _stack("stack_graph_768", "stack", 768, 768, blocks=4, graph=True),
        # The attention layers at 512 tokens, 475 of them valid.
        _attention("attention_512", 512, 475),
        # Throughput screening: a batch of 64 small proteins of 160 to 256 residues.
        _attention("attention_64x256", 256, 160, batch=64, transition=True),
        # The largest complex: one block of the row-chunked layers at 4096 tokens, 3900 valid.
        _attention("attention_4096", 4096, 3900, transition=True),
        # Unresolved residues inside the chain: a mask with holes, in its additive form.
        _attention("attention_holes_333", 333, 333, holes=True),
        # Triangle multiplication with its fp32 outputs (the constructor's default), odd and masked.
        {"name": "trimul_385", "kind": "trimul", "tokens": 385, "valid": 370, "batch": 1, "f32": True},
        # The ReLU pair transition with a mask.
        {"name": "transition_relu_640", "kind": "transition", "tokens": 640, "valid": 611, "batch": 1, "relu": True},
    ]


def _flops_cap():
    return max(work(c)["flops"] for c in listed())


def draw(rng):
    kind = rng.choice(["stack", "stack", "pair_stack", "attention", "attention", "attention", "trimul", "transition"])
    largest = {"stack": 800, "pair_stack": 800, "attention": 4096, "trimul": 2048, "transition": 2048}[kind]
    while True:
        tokens = round(math.exp(rng.uniform(math.log(24), math.log(largest))))
        case = {"kind": kind, "tokens": tokens, "valid": rng.choice([tokens, max(1, round(tokens * rng.uniform(0.6, 1.0)))])}
        case["batch"] = 1 if tokens > 1024 else rng.choice([1, 1, 2, 3, 8])
        if kind in ("stack", "pair_stack"):
            case.update(blocks=rng.choice([1, 2, 4]), graph=rng.random() < 0.5, f32=rng.random() < 0.3)
        elif kind == "attention":
            # the additive form of a mask is a tensor as large as the scores of one head: smaller proteins only
            case.update(transition=rng.random() < 0.5, holes=tokens <= 1024 and rng.random() < 0.2)
        elif kind == "trimul":
            case.update(f32=rng.random() < 0.5)
        else:
            case.update(relu=rng.random() < 0.5)
        if work(case)["flops"] <= _flops_cap() and case["batch"] * tokens * tokens <= 4096 * 4096:
            return case


# ---- inputs --------------------------------------------------------------------------------------------------------


def _lengths(case):
    n, valid, batch = case["tokens"], case["valid"], case["batch"]
    return [valid + (n - valid) * b // max(1, batch - 1) for b in range(batch)]


def _load(module, gen):
    """Trained-like weights: unit-variance projections, LayerNorm near the identity, small biases."""
    module = module.to("cuda")
    state = {}
    for key, p in module.state_dict().items():
        r = torch.randn(p.shape, generator=gen, device="cuda")
        if p.dim() == 2:
            r /= math.sqrt(p.shape[1])
        else:
            r = 0.1 * r + (0.0 if key.endswith("bias") else 1.0)
        state[key] = r.to(p.dtype)
    module.load_state_dict(state, strict=True)
    return module.eval()


def _token_mask(case, gen):
    n = case["tokens"]
    lengths = torch.tensor(_lengths(case), device="cuda")
    mask = (torch.arange(n, device="cuda")[None, :] < lengths[:, None]).float()
    if case.get("holes"):
        mask = mask * (torch.rand(mask.shape, generator=gen, device="cuda") > 0.1)
    return mask


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, batch, kind = case["tokens"], case["batch"], case["kind"]
    z = torch.randn(batch, n, n, C_Z, generator=gen, device="cuda", dtype=torch.bfloat16)
    mask = _token_mask(case, gen)
    pair_mask = mask[:, :, None] * mask[:, None, :]
    state = {"case": case, "z": z, "pair_mask": pair_mask, "buffers": {}}
    if kind in ("stack", "pair_stack"):
        options = dict(num_blocks=case["blocks"], dtype=torch.bfloat16, triangle_attn_backend="Heuristic",
                       trimul_high_precision=case["f32"], use_cuda_graph=case["graph"])
        if kind == "stack":
            module = b200.PairformerModule(token_s=C_S, num_heads=HEADS_S, attention_initial_norm=True, **options)
            state.update(s=torch.randn(batch, n, C_S, generator=gen, device="cuda", dtype=torch.bfloat16), mask=mask)
        else:
            module = b200.PairformerNoSeqModule(**options)
        state["stack"] = _load(module, gen)
    elif kind == "attention":
        backend = "VANILLA" if case["holes"] else "Heuristic"
        options = dict(dtype=torch.bfloat16, attn_backend=backend, pair_mask_left_aligned=not case["holes"])
        state["start"] = _load(b200.TriangleAttentionStartingNode(C_Z, 32, 4, **options), gen)
        state["end"] = _load(b200.TriangleAttentionEndingNode(C_Z, 32, 4, **options), gen)
        if case["transition"]:
            state["transition"] = _load(b200.Transition(C_Z, 4 * C_Z, dtype=torch.bfloat16), gen)
        state["masks"] = b200.precompute_pair_masks(backend, pair_mask)  # once per trunk, for all of its blocks
    elif kind == "trimul":
        types = b200.TriangleMultiplicationNodeType
        for name, direction in (("out", types.OUTGOING), ("in", types.INCOMING)):
            state[name] = _load(b200.TriangleMultiplicationNode(multiplication_type=direction, dtype=torch.bfloat16,
                                                                high_precision=case["f32"]), gen)
        masks = b200.precompute_pair_masks("Heuristic", pair_mask)
        state["metadata"] = b200.precompute_trimul_metadata(z, masks.mask_bias, masks.mask_bias_transposed)
    else:
        layer = (b200.PairTransition(C_Z, 4, dtype=torch.bfloat16) if case["relu"]
                 else b200.Transition(C_Z, 4 * C_Z, dtype=torch.bfloat16))
        state["transition"] = _load(layer, gen)
    return state


def run(state):
    kind, z = state["case"]["kind"], state["z"]
    if kind == "stack":
        return state["stack"](state["s"], z, state["mask"], state["pair_mask"])
    if kind == "pair_stack":
        return state["stack"](z, state["pair_mask"])
    if kind == "attention":
        masks, buffers = state["masks"], state["buffers"]
        z = state["start"](z, mask_bias=masks.mask_bias, buffers=buffers, residual=True)
        z = state["end"](z, mask_bias=masks.mask_bias_transposed, buffers=buffers, residual=True, inplace_residual=True)
        if state["case"]["transition"]:
            z = state["transition"](z, residual=True, inplace=True)
        return z
    if kind == "trimul":
        for node in (state["out"], state["in"]):
            z = node(z, state["pair_mask"], state["metadata"], residual=True, buffers=state["buffers"])
        return z
    return state["transition"](z, state["pair_mask"], residual=True)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------


def work(case):
    """The tensors read and written once; the operations on all positions, of the attention and of the contraction
    only those with valid keys (a pair row outside the valid tokens has no valid key)."""
    n, batch, kind = case["tokens"], case["batch"], case["kind"]
    lengths = [0.9 * v for v in _lengths(case)] if case.get("holes") else _lengths(case)
    positions = batch * n * n
    node = positions * 2 * C_Z * (4 * C_Z + 4 + C_Z) + sum(4 * C_Z * n * v * v for v in lengths)
    transition = positions * 2 * C_Z * 3 * 4 * C_Z
    trimul = positions * 2 * C_Z * 6 * C_Z + sum(2 * C_Z * v**3 for v in lengths)
    single = (positions * 2 * C_Z * HEADS_S + batch * n * 2 * C_S * C_S * (4 + 1 + 3 * 4)
              + sum(4 * C_S * n * v for v in lengths))
    weights = {"node": 2 * C_Z * (5 * C_Z + 4), "transition": 2 * C_Z * 12 * C_Z, "trimul": 2 * C_Z * 6 * C_Z,
               "single": 2 * (C_Z * HEADS_S + C_S * C_S * 17)}
    traffic = positions * 2 * C_Z * 2 + 4 * positions
    if kind in ("stack", "pair_stack"):
        block = 2 * node + 2 * trimul + transition
        held = 2 * weights["node"] + 2 * weights["trimul"] + weights["transition"]
        if kind == "stack":
            block, held, traffic = block + single, held + weights["single"], traffic + batch * n * C_S * 2 * 2
        return {"bytes": traffic + case["blocks"] * held, "flops": case["blocks"] * block}
    if kind == "attention":
        more = case["transition"]
        return {"bytes": traffic + 2 * weights["node"] + more * weights["transition"], "flops": 2 * node + more * transition}
    if kind == "trimul":
        wide = positions * C_Z * 2 if case["f32"] else 0  # the result in 4 bytes instead of 2
        return {"bytes": traffic + wide + 2 * weights["trimul"], "flops": 2 * trimul}
    if case["relu"]:
        return {"bytes": traffic + weights["transition"] * 2 // 3, "flops": transition * 2 // 3}
    return {"bytes": traffic + weights["transition"], "flops": transition}


def tolerance(case):
    # bfloat16 tensors between the layers: one rounding each in a layer, one per update of the residual stream in a stack
    deep = case.get("blocks", 1) > 2
    return {"rel": 2e-2 if deep else 1e-2, "max": 0.3 if deep else 0.15}
