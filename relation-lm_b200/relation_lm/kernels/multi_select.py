"""``relation_lm::relation_select_multi_rows`` / ``relation_select_multi_prefill`` — routed multi-anchor selection (extension).

The reference project's multi-anchor layer is dense: every slot scores all causal positions
(src/relation_lm/models/multi_relation_blocks.py:69-148).  This is its routed form, one launch
for all slots of every query row.  Its rules are the reference's, applied inside each slot's
routed candidate set (local window + that slot's best remote blocks):

* slot ``s`` is active for a query at position ``t`` iff ``s <= t``          (:82-84);
* slots choose their anchors one after another, a position taken by an earlier slot is barred
  (:86-93); an inactive slot reports anchor index 0                             (:94);
* partner selection of every slot bars the anchors of all active slots        (:133-139);
  an inactive slot has no partners                                            (:140-142);
* a partner slot is active iff its score is finite                            (:144-147).

With the window covering the whole history and no remote blocks the result equals the dense
block's selection (checked against outputs of the reference block itself).
"""
from __future__ import annotations

import torch
from torch import Tensor

from relation_lm.kernels import _abi  # noqa: F401  (loads the libraries)

# The operators themselves are registered by csrc/torch_ops.cpp; the functions below document them.
_relation_select_multi_rows = _abi.operator("relation_select_multi_rows")
_relation_select_multi_prefill = _abi.operator("relation_select_multi_prefill")
# the same without its last output (the partners' activity)
relation_select_multi_prefill_scores = _abi.operator("relation_select_multi_prefill_scores")
_slot_mix_residual = _abi.operator("slot_mix_residual")


def relation_select_multi_rows(
    anchor_query: Tensor,            # [N, S, 64]
    anchor_keys: Tensor,             # [S, B, T, 64]
    anchor_router_query: Tensor,     # [N, S, 64]
    anchor_block_mean: Tensor,       # [S, B, NB, 4, 16]
    anchor_block_std: Tensor,
    anchor_gamma: Tensor,            # [S, 4]
    anchor_bias: Tensor,             # [S, 4, buckets]
    partner_base: Tensor,            # [N, S, 128] query-side half of the factorised partner query
    partner_anchor_cache: Tensor,    # [S, B, T, 128] anchor-side half, cached per position
    partner_keys: Tensor,            # [S, B, T, 64]
    partner_block_mean: Tensor,
    partner_block_std: Tensor,
    partner_gamma: Tensor,
    partner_bias: Tensor,
    row_batch: Tensor,               # [N] int32
    row_position: Tensor,            # [N] int32
    local_window: int,
    top_blocks: int,
    partners_per_anchor: int,
    strict_valid: bool,
) -> tuple[Tensor, Tensor, Tensor, Tensor, Tensor, Tensor]:
    """Returns ``(anchor_index [N,S] i32, anchor_score [N,S], anchor_active [N,S] bool,
    partner_index [N,S,K] i32, partner_score [N,S,K], partner_active [N,S,K] bool)``."""
    return _relation_select_multi_rows(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean,
                                       anchor_block_std, anchor_gamma, anchor_bias, partner_base,
                                       partner_anchor_cache, partner_keys, partner_block_mean, partner_block_std,
                                       partner_gamma, partner_bias, row_batch, row_position, local_window,
                                       top_blocks, partners_per_anchor, strict_valid)


@torch.library.register_fake("relation_lm::relation_select_multi_rows")
def _(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean, anchor_block_std, anchor_gamma,
      anchor_bias, partner_base, partner_anchor_cache, partner_keys, partner_block_mean, partner_block_std,
      partner_gamma, partner_bias, row_batch, row_position, local_window, top_blocks, partners_per_anchor,
      strict_valid):
    rows, slots = anchor_query.size(0), anchor_query.size(1)
    k = partners_per_anchor
    f32 = torch.float32
    return (anchor_query.new_empty((rows, slots), dtype=torch.int32), anchor_query.new_empty((rows, slots), dtype=f32),
            anchor_query.new_empty((rows, slots), dtype=torch.bool),
            anchor_query.new_empty((rows, slots, k), dtype=torch.int32),
            anchor_query.new_empty((rows, slots, k), dtype=f32),
            anchor_query.new_empty((rows, slots, k), dtype=torch.bool))


def relation_select_multi_prefill(
    anchor_query: Tensor,            # [B * Tq, S, 64]
    anchor_keys: Tensor,             # [S, B, T, 64]
    anchor_router_query: Tensor,     # [B * Tq, S, 64]
    anchor_block_mean: Tensor,       # [S, B, NB, 4, 16]
    anchor_block_std: Tensor,
    anchor_gamma: Tensor,            # [S, 4]
    anchor_bias: Tensor,             # [S, 4, buckets]
    partner_base: Tensor,            # [B * Tq, S, 128]
    partner_anchor_cache: Tensor,    # [S, B, T, 128]
    partner_keys: Tensor,            # [S, B, T, 64]
    partner_block_mean: Tensor,
    partner_block_std: Tensor,
    partner_gamma: Tensor,
    partner_bias: Tensor,
    query_length: int,
    local_window: int,
    top_blocks: int,
    partners_per_anchor: int,
    strict_valid: bool,
) -> tuple[Tensor, Tensor, Tensor, Tensor, Tensor, Tensor]:
    """Whole-sequence form of ``relation_select_multi_rows`` (one 16-bit dtype throughout): query row
    ``b * query_length + t`` is position ``t`` of sequence ``b``; same results, bit for bit.  A CTA
    serves a tile of consecutive positions and stages each slot's block statistics and window union
    once per tile."""
    return _relation_select_multi_prefill(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean,
                                          anchor_block_std, anchor_gamma, anchor_bias, partner_base,
                                          partner_anchor_cache, partner_keys, partner_block_mean, partner_block_std,
                                          partner_gamma, partner_bias, query_length, local_window, top_blocks,
                                          partners_per_anchor, strict_valid)


@torch.library.register_fake("relation_lm::relation_select_multi_prefill")
def _(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean, anchor_block_std, anchor_gamma,
      anchor_bias, partner_base, partner_anchor_cache, partner_keys, partner_block_mean, partner_block_std,
      partner_gamma, partner_bias, query_length, local_window, top_blocks, partners_per_anchor, strict_valid):
    rows, slots = anchor_query.size(0), anchor_query.size(1)
    k = partners_per_anchor
    f32 = torch.float32
    return (anchor_query.new_empty((rows, slots), dtype=torch.int32), anchor_query.new_empty((rows, slots), dtype=f32),
            anchor_query.new_empty((rows, slots), dtype=torch.bool),
            anchor_query.new_empty((rows, slots, k), dtype=torch.int32),
            anchor_query.new_empty((rows, slots, k), dtype=f32),
            anchor_query.new_empty((rows, slots, k), dtype=torch.bool))


@torch.library.register_fake("relation_lm::relation_select_multi_prefill_scores")
def _(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean, anchor_block_std, anchor_gamma,
      anchor_bias, partner_base, partner_anchor_cache, partner_keys, partner_block_mean, partner_block_std,
      partner_gamma, partner_bias, query_length, local_window, top_blocks, partners_per_anchor, strict_valid):
    rows, slots = anchor_query.size(0), anchor_query.size(1)
    k = partners_per_anchor
    f32 = torch.float32
    return (anchor_query.new_empty((rows, slots), dtype=torch.int32), anchor_query.new_empty((rows, slots), dtype=f32),
            anchor_query.new_empty((rows, slots), dtype=torch.bool),
            anchor_query.new_empty((rows, slots, k), dtype=torch.int32),
            anchor_query.new_empty((rows, slots, k), dtype=f32))


def slot_mix_residual(slot_context: Tensor, anchor_active: Tensor, slot_weight: Tensor, gate: Tensor,
                      hidden: Tensor) -> None:
    """Last step of a multi-anchor layer (extension; multi_relation_blocks.py:170-178 of the reference):
    ``hidden += gate * sum_s w[:, s] * slot_context[:, s]`` with ``w`` the slot weights
    (``slot_weight [S]``, the softmax of the learned logits) renormalised over each row's active
    slots.  ``slot_context [N, S, d]``, ``hidden [N, d]``, ``gate`` (one element): fp32;
    ``anchor_active [N, S]`` bool."""
    _slot_mix_residual(slot_context, anchor_active, slot_weight, gate, hidden)


@torch.library.register_fake("relation_lm::slot_mix_residual")
def _(slot_context, anchor_active, slot_weight, gate, hidden):
    return None
