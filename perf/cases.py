"""What this framework is used for, as cases that can be timed: one relation layer's operators called
one by one, stateful decode (eager, as a captured graph, through the host loop, past the context), a
whole-sequence relation layer, and a multi-anchor stack over whole sequences.

A case is a dict of plain values.  ``listed()`` gives the standing ones, ``draw(rng)`` one more of the same
ranges; ``prepare(case, seed)`` builds what a program holds before the call, ``run(state)`` makes one pass
through the public entry points, ``work(case)`` counts the bytes and operations a pass cannot do without
and ``tolerance(case)`` says how far two correct implementations may be apart.
"""
from __future__ import annotations

import math
import os
import sys

_PACKAGE = os.path.join(os.getcwd(), "relation-lm_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(1, _PACKAGE)

import torch  # noqa: E402
import torch.nn.functional as F  # noqa: E402

from relation_lm.inference import pack_sparse_cache_projection_weights  # noqa: E402
from relation_lm.inference.multi_anchor import MultiAnchorConfig, MultiAnchorPrefill, MultiAnchorRoutedStack  # noqa: E402
from relation_lm.inference.prefill import RoutedPrefillLayer  # noqa: E402
from relation_lm.inference.routed_model import RoutedRelationConfig, RoutedRelationLM  # noqa: E402
from relation_lm.inference.stateful_decode import StatefulDecoder  # noqa: E402
from relation_lm.kernels.relation_reduce import (recommended_relation_cache_mode, relation_hidden_cache_update,  # noqa: E402
                                                 relation_hidden_cached, relation_norm_reduce)
from relation_lm.kernels.relation_select import relation_select_packed  # noqa: E402
from relation_lm.kernels.router_cache import router_cache_update  # noqa: E402

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
VOCAB, BOUNDARIES, R = 16_000, 256, 128


# ---------------------------------------------------------------------------- the cases


def _ops(name, dtype, batch, d_model, context, block, window, top, k, strict, position):
    return {"name": name, "kind": "ops", "dtype": dtype, "batch": batch, "d_model": d_model, "context": context,
            "block": block, "window": window, "top": top, "k": k, "strict": strict, "position": position}


def _decode(name, mode, dtype, batch, d_model, layers, context, block, window, top, start, steps):
    return {"name": name, "kind": "decode", "mode": mode, "dtype": dtype, "batch": batch, "d_model": d_model,
            "layers": layers, "context": context, "block": block, "window": window, "top": top, "start": start,
            "steps": steps}


def _prefill(name, dtype, batch, d_model, context, block, window, top, k, strict):
    return {"name": name, "kind": "prefill", "dtype": dtype, "batch": batch, "d_model": d_model, "context": context,
            "block": block, "window": window, "top": top, "k": k, "strict": strict}


def _multi(name, dtype, batch, d_model, context, block, window, top, slots, k, depth):
    return {"name": name, "kind": "multi", "dtype": dtype, "batch": batch, "d_model": d_model, "context": context,
            "block": block, "window": window, "top": top, "slots": slots, "k": k, "depth": depth}


def listed():
    return [
        # One decode position through the drop-in operators at the sizes and the routing policy the
        # reference project verifies (d 576, 512 positions, blocks of 8): the smallest call there is.
        _ops("ops fp32 batch 1", "fp32", 1, 576, 512, 8, 16, 2, 8, False, 476),
        # The same operators in 16 bits for a batch of requests, strict routing rule.
        _ops("ops bf16 batch 8", "bf16", 8, 576, 512, 8, 16, 1, 8, True, 500),
        # The single-layer model in single precision, stepped without a graph (debugging, evaluation).
        _decode("decode eager fp32", "eager", "fp32", 1, 256, 1, 128, 16, 32, 2, 100, 8),
        # One user of the 6-layer model: a captured step replayed over a piece of text.
        _decode("decode graph batch 1", "graph", "bf16", 1, 512, 6, 512, 32, 64, 2, 448, 32),
        # The serving loop of the 6-layer model: ids from the host and choices to the host at each position.
        _decode("decode host batch 8", "host", "bf16", 8, 512, 6, 512, 32, 64, 2, 448, 32),
        # A long generation by an odd number of users, its state sliding a block at a time.
        _decode("decode slide batch 5", "slide", "fp16", 5, 512, 6, 512, 32, 64, 2, 512, 32),
        # A GPU's share of the 256-sequence 12-layer job: many users, wide model, long context.
        _decode("decode graph batch 64", "graph", "bf16", 64, 768, 12, 2048, 64, 128, 2, 1000, 16),
        # A short prompt through one layer of a small model.
        _prefill("prefill small fp16", "fp16", 1, 256, 512, 16, 32, 2, 8, False),
        # Prompts of the wide model: an odd number of them, a context that fills no power of two.
        _prefill("prefill ragged d768", "bf16", 3, 768, 1984, 64, 128, 2, 8, True),
        # Long contexts: 8 sequences of 4096 positions.
        _prefill("prefill long", "bf16", 8, 512, 4096, 64, 128, 4, 8, False),
        # A shallow multi-anchor stack on a few sequences of uneven length.
        _multi("multi-anchor small", "bf16", 3, 256, 1056, 32, 64, 2, 2, 4, 2),
        # The multi-anchor stack of depth 4: 16 sequences, 4 anchors of 4 partners each.
        _multi("multi-anchor stack", "bf16", 16, 512, 2048, 32, 64, 3, 4, 4, 4),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.49))))))


def _blocks(rng, rows_low, rows_high, block):
    """A context length of whole blocks, spread over the logarithm of the range; at most 64 blocks."""
    rows = _log_int(rng, max(rows_low, 4 * block), min(rows_high, 64 * block))
    return max(4, rows // block) * block


def draw(rng):
    kind = rng.choice(("ops", "decode", "prefill", "multi"))
    if kind == "ops":
        dtype = rng.choice(("fp32", "bf16", "fp16"))
        block = rng.choice((8, 16, 32, 64))
        context = _blocks(rng, 128, 2048, block)
        window = rng.choice((16, 32, 48, 64))
        top = rng.randint(1, max(1, min(4, 128 // block)))
        case = _ops("", dtype, _log_int(rng, 1, 48), rng.choice((256, 512, 576, 768)), context, block, window, top,
                    rng.choice((4, 8)), rng.random() < 0.5, rng.randint(context // 2, context - 1))
    elif kind == "decode":
        mode = rng.choice(("eager", "graph", "host", "slide"))
        dtype = rng.choice(("fp32", "bf16", "bf16", "fp16"))
        sizes = ((256, 1), (256, 4), (512, 3), (512, 6), (768, 5), (768, 12))
        d_model, layers = rng.choice(sizes[:3] if mode == "eager" else sizes[:5] if mode == "slide" else sizes)
        block = rng.choice((16, 32) if mode == "slide" else (16, 32, 64))
        context = _blocks(rng, 256, 1024, block)
        batch = _log_int(rng, 1, 8 if dtype == "fp32" else 48)
        steps = block if mode == "slide" else rng.randint(2, 6) if mode == "eager" else rng.randint(4, 16)
        start = context if mode == "slide" else rng.randint(context // 2, context - steps)
        case = _decode("", mode, dtype, batch, d_model, layers, context, block, rng.choice((32, 64)),
                       rng.randint(1, 2), start, steps)
    elif kind == "prefill":
        d_model = rng.choice((256, 512, 768))
        block = rng.choice((16, 32, 64))
        context = _blocks(rng, 256, 4096, block)
        batch = _log_int(rng, 1, max(1, min(9, 24_576 // context)))
        case = _prefill("", rng.choice(("bf16", "bf16", "fp16")), batch, d_model, context, block,
                        rng.choice((32, 64, 128)), rng.randint(1, 4), rng.choice((4, 8)), rng.random() < 0.5)
    else:
        d_model = rng.choice((256, 512))
        block = rng.choice((16, 32, 64))
        context = _blocks(rng, 256, 2048, block)
        batch = _log_int(rng, 1, max(1, min(9, 12_288 // context)))
        case = _multi("", rng.choice(("bf16", "bf16", "fp16")), batch, d_model, context, block, rng.choice((32, 64)),
                      rng.randint(1, 3), rng.randint(2, 4), rng.choice((4, 8)), rng.randint(1, 3))
    del case["name"]
    return case


# ---------------------------------------------------------------------------- inputs


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _hidden_states(g, batch, context, d_model):
    """N(0, 1) rows of which one in twenty is four times as large: strong anchors."""
    x = torch.randn(batch, context, d_model, generator=g, device="cuda")
    strong = torch.rand(batch, context, 1, generator=g, device="cuda") < 0.05
    return torch.where(strong, 4.0 * x, x)


def _text(g, positions, batch):
    """Token ids bounded Zipf(1.1) over the vocabulary, boundary ids uniform: ``[positions, batch]`` each."""
    weights = torch.arange(1, VOCAB + 1, device="cuda", dtype=torch.float32).pow(-1.1)
    tokens = torch.multinomial(weights, positions * batch, replacement=True, generator=g).view(positions, batch)
    bounds = torch.randint(0, BOUNDARIES, (positions, batch), generator=g, device="cuda")
    return tokens, bounds


def _prepare_ops(c, seed):
    g = _generator(seed)
    dtype, B, d, T = DTYPES[c["dtype"]], c["batch"], c["d_model"], c["context"]
    H, NB = 4 * d, c["context"] // c["block"]
    linear = lambda n, k: _randn(g, n, k, dtype=dtype, scale=(2.0 / (n + k)) ** 0.5)  # noqa: E731
    s = {"case": c, "dtype": dtype, "memory": _randn(g, B, d, dtype=dtype),
         "projection": pack_sparse_cache_projection_weights([linear(n, d) for n in (64, 64, R, 128, 64, 64)]),
         "anchor_query": _randn(g, B, 64, dtype=dtype), "anchor_router_query": _randn(g, B, 64, dtype=dtype),
         "partner_base": _randn(g, B, 128, dtype=dtype), "anchor_keys": _randn(g, B, T, 64, dtype=dtype),
         "partner_keys": _randn(g, B, T, 64, dtype=dtype), "partner_anchor_cache": _randn(g, B, T, 128, dtype=dtype),
         "operand_cache": _randn(g, B, T, R, dtype=dtype), "expanded_cache": _randn(g, B, T, 2 * H, dtype=dtype, scale=0.3),
         "anchor_gamma": _randn(g, 4), "anchor_bias": _randn(g, 4, 16), "partner_gamma": _randn(g, 4),
         "partner_bias": _randn(g, 4, 16), "anchor_conv": _randn(g, 64, 3, scale=0.1),
         "partner_conv": _randn(g, 64, 3, scale=0.1),
         "anchor_weight": linear(H, R), "partner_weight": linear(H, R), "product_weight": linear(H, R),
         "first_bias": _randn(g, H, dtype=dtype, scale=0.02), "w2": linear(d, H), "b2": _randn(g, d, dtype=dtype, scale=0.02),
         "norm_weight": 1.0 + _randn(g, d, scale=0.05), "norm_bias": _randn(g, d, scale=0.05),
         "position": torch.tensor(c["position"], device="cuda", dtype=torch.int64)}
    s["expanded_weight"] = torch.cat((s["anchor_weight"], s["partner_weight"]), 0)
    s["expanded_bias"] = torch.cat((s["first_bias"], torch.zeros_like(s["first_bias"])), 0)
    s["router"] = [_randn(g, B, T, 64, dtype=dtype) for _ in range(4)]
    s["statistics"] = [_randn(g, B, NB, 4, 16, dtype=dtype), _randn(g, B, NB, 4, 16, dtype=dtype).abs(),
                       _randn(g, B, NB, 4, 16, dtype=dtype), _randn(g, B, NB, 4, 16, dtype=dtype).abs()]
    return s


def _prepare_decode(c, seed):
    g = _generator(seed)
    cfg = RoutedRelationConfig(vocab_size=VOCAB, boundary_vocab_size=BOUNDARIES, d_model=c["d_model"], layers=c["layers"],
                               max_context=c["context"], block_size=c["block"], local_window=c["window"],
                               top_blocks=c["top"])
    dec = StatefulDecoder(RoutedRelationLM(cfg, seed=seed), c["batch"], "cuda", DTYPES[c["dtype"]])
    # the prompt: the decoder reads it as it reads everything, a position at a time
    tokens, bounds = _text(g, c["start"], c["batch"])
    dec.capture()
    for i in range(c["start"]):
        dec.static_tokens.copy_(tokens[i])
        dec.static_boundaries.copy_(bounds[i])
        dec.replay()
    if c["mode"] == "host":
        dec.capture_host_io()
    tokens, bounds = _text(g, c["steps"], c["batch"])
    if c["mode"] == "host":
        tokens, bounds = tokens.cpu(), bounds.cpu()
    return {"case": c, "decoder": dec, "tokens": tokens, "bounds": bounds,
            "chosen": torch.zeros(c["steps"], c["batch"], dtype=torch.int64, device=tokens.device)}


def _prepare_prefill(c, seed):
    cfg = RoutedRelationConfig(vocab_size=64, boundary_vocab_size=8, d_model=c["d_model"], layers=1,
                               max_context=c["context"], block_size=c["block"], local_window=c["window"],
                               top_blocks=c["top"], k_max=c["k"], strict_valid=c["strict"])
    layer = RoutedPrefillLayer(RoutedRelationLM(cfg, seed=seed), 0, "cuda", DTYPES[c["dtype"]])
    return {"case": c, "layer": layer, "x": _hidden_states(_generator(seed), c["batch"], c["context"], c["d_model"])}


def _prepare_multi(c, seed):
    cfg = MultiAnchorConfig(d_model=c["d_model"], anchors_per_block=c["slots"], partners_per_anchor=c["k"],
                            depth=c["depth"], max_context=c["context"], block_size=c["block"],
                            local_window=c["window"], top_blocks=c["top"])
    dtype, g = DTYPES[c["dtype"]], _generator(seed)
    stack = MultiAnchorPrefill(MultiAnchorRoutedStack(cfg, seed=seed), "cuda", dtype)
    return {"case": c, "stack": stack, "hidden": _randn(g, c["batch"], c["context"], c["d_model"]),
            "memory": _randn(g, c["batch"], c["context"], c["d_model"], dtype=dtype)}


def prepare(case, seed):
    return {"ops": _prepare_ops, "decode": _prepare_decode, "prefill": _prepare_prefill,
            "multi": _prepare_multi}[case["kind"]](case, seed)


# ---------------------------------------------------------------------------- one pass


def _run_ops(s):
    """A position of one layer: project the memory row, update the router state, select, and reduce the
    selected relations, with the expanded cache kept as the library recommends for the batch."""
    c, pos = s["case"], s["position"]
    parts = s["projection"].project(s["memory"])
    conv = router_cache_update(parts[4], parts[5], *s["router"], *s["statistics"], s["anchor_conv"], s["partner_conv"],
                               pos, c["block"])
    mean_a, std_a, mean_p, std_p = s["statistics"]
    anchor, anchor_score, partner, score = relation_select_packed(
        s["anchor_query"], s["anchor_keys"], s["anchor_router_query"], mean_a, std_a, s["anchor_gamma"], s["anchor_bias"],
        s["partner_base"], s["partner_anchor_cache"], s["partner_keys"], mean_p, std_p, s["partner_gamma"],
        s["partner_bias"], pos, c["window"], c["top"], c["k"], c["strict"])
    if recommended_relation_cache_mode(c["batch"]) == "fused_update":
        hidden = relation_hidden_cache_update(s["expanded_cache"], s["operand_cache"], anchor, partner, s["anchor_weight"],
                                              s["partner_weight"], s["product_weight"], s["first_bias"], pos)
    else:
        row = F.linear(parts[2], s["expanded_weight"], s["expanded_bias"])
        s["expanded_cache"].index_copy_(1, pos.view(1), row.unsqueeze(1))
        hidden = relation_hidden_cached(s["expanded_cache"], s["operand_cache"], anchor, partner, s["product_weight"])
    raw = F.linear(hidden.to(s["dtype"]), s["w2"], s["b2"])
    context = relation_norm_reduce(raw, score, s["norm_weight"], s["norm_bias"], pos, 1.0e-5)
    return [list(parts), conv, anchor, anchor_score, partner, score, hidden, raw, context, s["router"], s["statistics"],
            s["expanded_cache"]]


def _run_decode(s):
    """A piece of text at the end of the prompt, a position at a time."""
    c, dec, tokens, bounds, chosen = s["case"], s["decoder"], s["tokens"], s["bounds"], s["chosen"]
    if c["mode"] == "slide":
        dec.slide(1)
    else:
        dec.position.fill_(c["start"])
    if c["mode"] == "eager":
        logits = []
        for i in range(c["steps"]):
            logits.append(torch.cat(dec.step(tokens[i], bounds[i]), 1))
        logits, chosen = torch.stack(logits), None
    elif c["mode"] == "host":
        for i in range(c["steps"]):
            dec.host_tokens.copy_(tokens[i])
            dec.host_boundaries.copy_(bounds[i])
            chosen[i].copy_(dec.step_host())
        logits = dec.last_logits if dec.fused else None
    else:
        for i in range(c["steps"]):
            dec.static_tokens.copy_(tokens[i])
            dec.static_boundaries.copy_(bounds[i])
            dec.replay()
            chosen[i].copy_(dec.static_next)
        logits = [dec.static_token_logits, dec.static_boundary_logits]
    return [chosen, logits, dec.position, dec.anchor_keys, dec.partner_keys, dec.operand_cache, dec.partner_anchor_cache,
            list(dec.expanded_cache), dec.router_caches, dec.router_stats]


def _run_prefill(s):
    state = s["layer"].build_state(s["x"])
    return [s["layer"].forward(s["x"], state), state]


def _run_multi(s):
    return s["stack"].forward(s["hidden"], s["memory"])


def run(state):
    return {"ops": _run_ops, "decode": _run_decode, "prefill": _run_prefill,
            "multi": _run_multi}[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------- what a pass cannot do without


def _selection(c, e, rows, complete_blocks):
    """Bytes and operations of one layer's (or slot's) selection for ``rows`` queries, each with history of its own."""
    cand = c["window"] + c["top"] * c["block"]
    size = rows * (e * (4 * complete_blocks * 64 + 2 * cand * 64 + 384) + 560 + 8 + 8 * c.get("k", 8))
    return size, rows * 2 * (2 * cand * 64 + 2 * 2 * complete_blocks * 64)


def _work_ops(c):
    e, B, d, K, H = (4 if c["dtype"] == "fp32" else 2), c["batch"], c["d_model"], c["k"], 4 * c["d_model"]
    size, flops = _selection(c, e, B, c["position"] // c["block"])
    size += e * (B * d + 512 * d + B * 512)                                       # packed projection
    size += B * (e * 64 * (14 + 2 * c["block"]) + 512)                            # router state
    size += e * (3 * H * R + B * R + 2 * B * H)                                   # the position's expanded row
    size += B * (e * (1 + K) * (H + R) + 4 * K * H)                               # hidden states
    size += e * (H * d + B * K * d) + B * (4 * K + 4 * d) + 8 * d                 # second layer, norm, reduction
    flops += 2 * B * (512 * d + 2 * H * R + K * (H * R + H * d))
    return size, flops


def _work_decode(c):
    e, B, d, L, K = (4 if c["dtype"] == "fp32" else 2), c["batch"], c["d_model"], c["layers"], 8
    H, heads = 4 * d, VOCAB + BOUNDARIES
    blocks = min(c["start"], c["context"] - 1) // c["block"]
    size, flops = _selection(c, e, B, blocks)
    size += e * d * (512 + 256 + H) + 3 * e * H * R                               # a layer's weights
    size += B * (e * (768 + 64 * (14 + 2 * c["block"]) + 2 * H) + e * (1 + K) * (H + R) + 8 * d)
    flops += 2 * B * (d * (512 + 256) + 2 * H * R + K * (H * R + H * d))
    size, flops = L * size + e * d * heads + B * (e * heads + 2 * e * d), L * flops + 2 * B * d * heads
    size, flops = c["steps"] * size, c["steps"] * flops
    if c["mode"] == "slide":
        row = L * B * e * (64 + 64 + R + 128 + 2 * H + 4 * 64 + 4 * 64 / c["block"])
        size += 2 * row * (c["context"] - c["block"])
    return size, flops


def _work_prefill(c):
    e, N, d, K, H = 2, c["batch"] * c["context"], c["d_model"], c["k"], 4 * c["d_model"]
    nb = c["context"] // c["block"]
    size = 4 * N * d + e * d * (512 + 256 + H) + 3 * e * H * R + 4 * N * d        # rows in, weights, rows out
    size += e * N * (512 + 384 + 2 * 64 * 2 + 2 * H) + 4 * e * c["batch"] * nb * 64    # the state: written once
    size += e * N * (64 + 64 + 128 + R + 2 * H)                                   # ... and read once by the layer
    cand = c["window"] + c["top"] * c["block"]
    flops = N * 2 * (2 * cand * 64 + 2 * nb * 64)
    flops += 2 * N * (d * (512 + 256) + 2 * H * R + K * (H * R + H * d))
    return size, flops


def _work_multi(c):
    e, N, d, S, K, H = 2, c["batch"] * c["context"], c["d_model"], c["slots"], c["k"], 4 * c["d_model"]
    nb, cand = c["context"] // c["block"], c["window"] + c["top"] * c["block"]
    size = (4 + e + 8) * N * d + e * d * (S * (384 + 256) + R + H) + 3 * e * H * R
    flops = N * S * 2 * (2 * cand * 64 + 2 * nb * 64)
    flops += 2 * N * (d * (S * (384 + 256) + R) + 2 * H * R + S * K * (H * R + H * d))
    return c["depth"] * size, c["depth"] * flops


def work(case):
    size, flops = {"ops": _work_ops, "decode": _work_decode, "prefill": _work_prefill,
                   "multi": _work_multi}[case["kind"]](case)
    return {"bytes": float(size), "flops": float(flops)}


def tolerance(case):
    """Single precision: the order of the sums.  16 bits: the rounding of the layers' intermediates, and
    selections that fall the other way where two scores agree to that rounding (a row's result then moves
    by up to its gate times a context, which ``max`` allows for)."""
    if case["dtype"] == "fp32":
        return {"rel": 1.0e-5, "max": 1.0e-3, "differ": 0.0}
    return {"rel": 1.0e-2, "max": 0.99, "differ": 0.01}
