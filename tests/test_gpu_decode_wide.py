"""16-bit decoders on the routes that their size chooses: d 768 with the relation layer tail and without, and more than 16
sequences, whose expanded rows are made from the packed rows while the cache append is under way."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear

pytestmark = pytest.mark.gpu

STATE = ("anchor_keys", "partner_keys", "operand_cache", "partner_anchor_cache", "expanded_cache")


def _model(d_model, layers, seed, **kw):
    from relation_lm.inference.routed_model import RoutedRelationConfig, RoutedRelationLM

    cfg = RoutedRelationConfig(vocab_size=500, boundary_vocab_size=16, d_model=d_model, layers=layers, max_context=48, block_size=8,
                               local_window=16, top_blocks=2, **kw)
    return RoutedRelationLM(cfg, seed=seed)


def _ids(batch, steps, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(0, 500, (steps, batch), generator=g).cuda(), torch.randint(0, 16, (steps, batch), generator=g).cuda()


def _same_state(one, two):
    for name in STATE:
        assert torch.equal(getattr(one, name), getattr(two, name)), name
    for a, b in zip(one.router_caches + one.router_stats, two.router_caches + two.router_stats):
        assert torch.equal(a, b)


@pytest.mark.parametrize("batch,k,dtype,tail", [
    (1, 8, torch.bfloat16, True), (8, 8, torch.float16, True), (31, 8, torch.bfloat16, True), (60, 4, torch.bfloat16, True),
    (32, 8, torch.bfloat16, False), (33, 8, torch.float16, False)])
def test_wide_step_eager_captured_and_past_the_context(batch, k, dtype, tail):
    """With and without programmatic launch and replayed from a graph, sliding once: the same bits; beside the route that
    was not chosen: the same selections but for rare near-ties, logits within 16-bit noise."""
    from relation_lm.inference.stateful_decode import StatefulDecoder

    model = _model(768, 2, batch, k_max=k)
    plain = StatefulDecoder(model, batch, "cuda", dtype, programmatic_launch=False)
    early = StatefulDecoder(model, batch, "cuda", dtype)
    graphed = StatefulDecoder(model, batch, "cuda", dtype)
    other = StatefulDecoder(model, batch, "cuda", dtype, layer_tail=not tail)
    assert plain.layer_tail == early.layer_tail == graphed.layer_tail == tail and other.layer_tail != tail
    graphed.capture()
    tokens, bounds = _ids(batch, 56, batch)
    agree = total = 0
    for t in range(56):
        if t == 48:
            for dec in (plain, early, graphed, other):
                dec.slide(1)
        a = plain.step(tokens[t], bounds[t], keep_selection=True)
        b = early.step(tokens[t], bounds[t], keep_selection=True)
        c = other.step(tokens[t], bounds[t], keep_selection=True)
        graphed.static_tokens.copy_(tokens[t])
        graphed.static_boundaries.copy_(bounds[t])
        graphed.replay()
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1]), t
        assert torch.equal(a[0], graphed.static_token_logits) and torch.equal(a[1], graphed.static_boundary_logits), t
        same = torch.ones(batch, dtype=torch.bool, device="cuda")
        for (anchor, partner), (other_anchor, other_partner) in zip(plain.last_selection, other.last_selection):
            same &= (anchor == other_anchor).view(batch, -1).all(1) & (partner == other_partner).view(batch, -1).all(1)
        agree, total = agree + int(same.sum()), total + batch
        assert torch.allclose(a[0][same].float(), c[0][same].float(), atol=0.25, rtol=0.05), t
    assert agree >= 0.9 * total
    _same_state(plain, early)
    _same_state(plain, graphed)
    assert_status_clear()


@pytest.mark.parametrize("batch,d_model,dtype", [(17, 128, torch.bfloat16), (24, 256, torch.bfloat16), (32, 512, torch.float16),
                                                 (70, 256, torch.bfloat16)])
def test_expanded_rows_made_beside_the_cache_append(batch, d_model, dtype):
    """Every expanded row is what the operator makes of the operand cache, and the launches that overlap change nothing."""
    from relation_lm.inference.stateful_decode import StatefulDecoder
    from relation_lm.kernels.relation_reduce import expanded_cache_append

    model = _model(d_model, 3, batch)
    plain = StatefulDecoder(model, batch, "cuda", dtype, programmatic_launch=False)
    early = StatefulDecoder(model, batch, "cuda", dtype)
    graphed = StatefulDecoder(model, batch, "cuda", dtype)
    assert early.stacked_expand and not early.fused_front and not early.append_in_projection
    graphed.capture()
    tokens, bounds = _ids(batch, 24, batch)
    want = torch.zeros_like(early.expanded_cache)
    for t in range(24):
        a, b = plain.step(tokens[t], bounds[t]), early.step(tokens[t], bounds[t])
        graphed.static_tokens.copy_(tokens[t])
        graphed.static_boundaries.copy_(bounds[t])
        graphed.replay()
        assert torch.equal(a[0], b[0]) and torch.equal(a[0], graphed.static_token_logits), t
        w = early.w
        expanded_cache_append(want, early.operand_cache, w["anchor_weight"], w["partner_weight"], w["first_bias"],
                              torch.tensor(t, device="cuda"))
    assert torch.equal(early.expanded_cache, want)
    _same_state(plain, early)
    _same_state(plain, graphed)
    assert_status_clear()
