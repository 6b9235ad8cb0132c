"""``relation_lm::relation_select_packed`` — fused routed anchor/partner selection.

Same operator name, schema and semantics as the reference project's
``src/relation_lm/kernels/relation_select.py:311-382`` (compatibility and
strict-valid remote-block rules included); the body is one launch of the
sm_100a kernel ``relation_select_kernel`` through the C ABI.
``relation_select_packed_rows`` is an additive extension for query rows that
carry their own sequence index and position (prefill).
"""
from __future__ import annotations

import torch
from torch import Tensor

from relation_lm.kernels import _abi  # noqa: F401  (loads the libraries)

# The operators themselves are registered by csrc/torch_ops.cpp; the functions below document them.
_relation_select_packed = _abi.operator("relation_select_packed")
_relation_select_packed_rows = _abi.operator("relation_select_packed_rows")
_relation_select_packed_prefill = _abi.operator("relation_select_packed_prefill")


def relation_select_packed(
    anchor_query: Tensor,
    anchor_keys: Tensor,
    anchor_router_query: Tensor,
    anchor_block_mean: Tensor,
    anchor_block_std: Tensor,
    anchor_gamma: Tensor,
    anchor_bias: Tensor,
    partner_base: Tensor,
    partner_anchor_cache: Tensor,
    partner_keys: Tensor,
    partner_block_mean: Tensor,
    partner_block_std: Tensor,
    partner_gamma: Tensor,
    partner_bias: Tensor,
    position: Tensor,
    local_window: int,
    top_blocks: int,
    k_out: int,
    strict_valid: bool,
) -> tuple[Tensor, Tensor, Tensor, Tensor]:
    """Anchor index/score ``[B]`` and partner indices/scores ``[B, k_out]`` at ``position``."""
    return _relation_select_packed(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean,
                                   anchor_block_std, anchor_gamma, anchor_bias, partner_base, partner_anchor_cache,
                                   partner_keys, partner_block_mean, partner_block_std, partner_gamma, partner_bias,
                                   position, local_window, top_blocks, k_out, strict_valid)


@torch.library.register_fake("relation_lm::relation_select_packed")
def _(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean, anchor_block_std,
      anchor_gamma, anchor_bias, partner_base, partner_anchor_cache, partner_keys,
      partner_block_mean, partner_block_std, partner_gamma, partner_bias, position, local_window,
      top_blocks, k_out, strict_valid):
    rows = anchor_query.size(0)
    return (anchor_query.new_empty((rows,), dtype=torch.int32),
            anchor_query.new_empty((rows,), dtype=torch.float32),
            anchor_query.new_empty((rows, k_out), dtype=torch.int32),
            anchor_query.new_empty((rows, k_out), dtype=torch.float32))


def relation_select_packed_rows(
    anchor_query: Tensor,
    anchor_keys: Tensor,
    anchor_router_query: Tensor,
    anchor_block_mean: Tensor,
    anchor_block_std: Tensor,
    anchor_gamma: Tensor,
    anchor_bias: Tensor,
    partner_base: Tensor,
    partner_anchor_cache: Tensor,
    partner_keys: Tensor,
    partner_block_mean: Tensor,
    partner_block_std: Tensor,
    partner_gamma: Tensor,
    partner_bias: Tensor,
    row_batch: Tensor,
    row_position: Tensor,
    local_window: int,
    top_blocks: int,
    k_out: int,
    strict_valid: bool,
) -> tuple[Tensor, Tensor, Tensor, Tensor]:
    """Per-row form: query row ``i`` selects in sequence ``row_batch[i]`` at ``row_position[i]``.

    Row ``i`` equals ``relation_select_packed`` called with ``position = row_position[i]`` on
    that sequence, given block statistics that are final for every complete block.
    """
    return _relation_select_packed_rows(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean,
                                        anchor_block_std, anchor_gamma, anchor_bias, partner_base,
                                        partner_anchor_cache, partner_keys, partner_block_mean, partner_block_std,
                                        partner_gamma, partner_bias, row_batch, row_position, local_window,
                                        top_blocks, k_out, strict_valid)


@torch.library.register_fake("relation_lm::relation_select_packed_rows")
def _(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean, anchor_block_std,
      anchor_gamma, anchor_bias, partner_base, partner_anchor_cache, partner_keys,
      partner_block_mean, partner_block_std, partner_gamma, partner_bias, row_batch, row_position,
      local_window, top_blocks, k_out, strict_valid):
    rows = anchor_query.size(0)
    return (anchor_query.new_empty((rows,), dtype=torch.int32),
            anchor_query.new_empty((rows,), dtype=torch.float32),
            anchor_query.new_empty((rows, k_out), dtype=torch.int32),
            anchor_query.new_empty((rows, k_out), dtype=torch.float32))


def relation_select_packed_prefill(
    anchor_query: Tensor,
    anchor_keys: Tensor,
    anchor_router_query: Tensor,
    anchor_block_mean: Tensor,
    anchor_block_std: Tensor,
    anchor_gamma: Tensor,
    anchor_bias: Tensor,
    partner_base: Tensor,
    partner_anchor_cache: Tensor,
    partner_keys: Tensor,
    partner_block_mean: Tensor,
    partner_block_std: Tensor,
    partner_gamma: Tensor,
    partner_bias: Tensor,
    query_length: int,
    local_window: int,
    top_blocks: int,
    k_out: int,
    strict_valid: bool,
) -> tuple[Tensor, Tensor, Tensor, Tensor]:
    """Whole-sequence form (extension): the queries are rows ``b * query_length + t`` for every
    position ``t < query_length`` of every sequence ``b`` of caches ``[B, T, ...]``; row ``(b, t)``
    equals ``relation_select_packed`` at ``position = t`` on sequence ``b`` (given final block
    statistics), bit for bit.  A CTA serves a tile of consecutive positions: their shared block
    statistics and the union of their local windows are staged once, and every warp walks one
    query's chain at a time.  At most 512 candidates per query (window + remote blocks)."""
    return _relation_select_packed_prefill(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean,
                                           anchor_block_std, anchor_gamma, anchor_bias, partner_base,
                                           partner_anchor_cache, partner_keys, partner_block_mean, partner_block_std,
                                           partner_gamma, partner_bias, query_length, local_window, top_blocks,
                                           k_out, strict_valid)


@torch.library.register_fake("relation_lm::relation_select_packed_prefill")
def _(anchor_query, anchor_keys, anchor_router_query, anchor_block_mean, anchor_block_std, anchor_gamma,
      anchor_bias, partner_base, partner_anchor_cache, partner_keys, partner_block_mean, partner_block_std,
      partner_gamma, partner_bias, query_length, local_window, top_blocks, k_out, strict_valid):
    rows = anchor_query.size(0)
    return (anchor_query.new_empty((rows,), dtype=torch.int32), anchor_query.new_empty((rows,), dtype=torch.float32),
            anchor_query.new_empty((rows, k_out), dtype=torch.int32),
            anchor_query.new_empty((rows, k_out), dtype=torch.float32))
