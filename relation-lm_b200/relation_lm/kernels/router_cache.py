"""``relation_lm::router_cache_update`` — stateful router-key update for one position.

Same operator name, schema and mutated arguments as the reference project's
``src/relation_lm/kernels/router_cache.py:175-241``; one launch of the sm_100a
kernel ``router_cache_update_kernel`` through the C ABI.
"""
from __future__ import annotations

import torch
from torch import Tensor

from relation_lm.kernels import _abi

# The operators themselves are registered by csrc/torch_ops.cpp; the functions below document them.
_router_cache_update = _abi.operator("router_cache_update")
_sparse_cache_append = _abi.operator("sparse_cache_append")
_sequence_state = _abi.operator("sequence_state")
_router_cache_prefill = _abi.operator("router_cache_prefill")

_MUTATED = ("anchor_raw_cache", "partner_raw_cache", "anchor_conv_cache", "partner_conv_cache",
            "anchor_mean", "anchor_std", "partner_mean", "partner_std")


def router_cache_update(
    anchor_raw: Tensor,
    partner_raw: Tensor,
    anchor_raw_cache: Tensor,
    partner_raw_cache: Tensor,
    anchor_conv_cache: Tensor,
    partner_conv_cache: Tensor,
    anchor_mean: Tensor,
    anchor_std: Tensor,
    partner_mean: Tensor,
    partner_std: Tensor,
    anchor_conv_weight: Tensor,
    partner_conv_weight: Tensor,
    position: Tensor,
    block_size: int,
) -> Tensor:
    """Write raw and causally convolved router keys at ``position`` and refresh that block's
    mean / biased std for both streams.  ``anchor_raw`` / ``partner_raw`` may be column slices
    of a wider packed projection (row stride is honoured, inner stride must be 1).
    Returns the convolved keys ``[B, 2, 64]`` in fp32."""
    return _router_cache_update(anchor_raw, partner_raw, anchor_raw_cache, partner_raw_cache, anchor_conv_cache,
                                partner_conv_cache, anchor_mean, anchor_std, partner_mean, partner_std,
                                anchor_conv_weight, partner_conv_weight, position, block_size)


@torch.library.register_fake("relation_lm::router_cache_update")
def _(anchor_raw, partner_raw, anchor_raw_cache, partner_raw_cache, anchor_conv_cache,
      partner_conv_cache, anchor_mean, anchor_std, partner_mean, partner_std,
      anchor_conv_weight, partner_conv_weight, position, block_size):
    return anchor_raw.new_empty((anchor_raw.size(0), 2, anchor_raw.size(1)), dtype=torch.float32)


_APPEND_MUTATED = ("anchor_keys", "partner_keys", "operand_cache", "partner_anchor_cache") + _MUTATED


def sparse_cache_append(
    packed: Tensor,
    anchor_keys: Tensor,
    partner_keys: Tensor,
    operand_cache: Tensor,
    partner_anchor_cache: Tensor,
    anchor_raw_cache: Tensor,
    partner_raw_cache: Tensor,
    anchor_conv_cache: Tensor,
    partner_conv_cache: Tensor,
    anchor_mean: Tensor,
    anchor_std: Tensor,
    partner_mean: Tensor,
    partner_std: Tensor,
    anchor_conv_weight: Tensor,
    partner_conv_weight: Tensor,
    position: Tensor,
    block_size: int,
) -> None:
    """All layers of a stack at once: write the packed projection's token features into row
    ``position`` of their caches and update both router streams (extension of
    ``router_cache_update``; every cache carries a leading layer dimension and ``packed`` is
    ``[B, layers * (384 + R)]`` in the packed column order)."""
    _sparse_cache_append(packed, anchor_keys, partner_keys, operand_cache, partner_anchor_cache, anchor_raw_cache,
                         partner_raw_cache, anchor_conv_cache, partner_conv_cache, anchor_mean, anchor_std,
                         partner_mean, partner_std, anchor_conv_weight, partner_conv_weight, position, block_size)


@torch.library.register_fake("relation_lm::sparse_cache_append")
def _(packed, anchor_keys, partner_keys, operand_cache, partner_anchor_cache, anchor_raw_cache,
      partner_raw_cache, anchor_conv_cache, partner_conv_cache, anchor_mean, anchor_std,
      partner_mean, partner_std, anchor_conv_weight, partner_conv_weight, position, block_size):
    return None


def router_cache_prefill(
    anchor_raw: Tensor,
    partner_raw: Tensor,
    anchor_raw_cache: Tensor,
    partner_raw_cache: Tensor,
    anchor_conv_cache: Tensor,
    partner_conv_cache: Tensor,
    anchor_mean: Tensor,
    anchor_std: Tensor,
    partner_mean: Tensor,
    partner_std: Tensor,
    anchor_conv_weight: Tensor,
    partner_conv_weight: Tensor,
    block_size: int,
) -> None:
    """Fill zero-initialised router caches and block statistics for a whole prefix
    ``anchor_raw, partner_raw [B, length, 64]`` in one launch (extension); the state equals that
    of ``length`` successive ``router_cache_update`` calls."""
    _router_cache_prefill(anchor_raw, partner_raw, anchor_raw_cache, partner_raw_cache, anchor_conv_cache,
                          partner_conv_cache, anchor_mean, anchor_std, partner_mean, partner_std, anchor_conv_weight,
                          partner_conv_weight, block_size)


@torch.library.register_fake("relation_lm::router_cache_prefill")
def _(anchor_raw, partner_raw, anchor_raw_cache, partner_raw_cache, anchor_conv_cache,
      partner_conv_cache, anchor_mean, anchor_std, partner_mean, partner_std,
      anchor_conv_weight, partner_conv_weight, block_size):
    return None


STATE_NAMES = ("anchor_keys", "partner_keys", "operand_cache", "partner_anchor_cache", "anchor_raw_cache",
               "partner_raw_cache", "anchor_conv_cache", "partner_conv_cache", "anchor_mean", "anchor_std",
               "partner_mean", "partner_std")


def sequence_state(packed: Tensor, slots: int, relation_dim: int, block_size: int, anchor_conv_weight: Tensor,
                   partner_conv_weight: Tensor) -> dict[str, Tensor]:
    """The memory-side state of whole sequences from their packed projection rows ``[B, T, W]`` (16-bit) in one
    launch (extension), keyed by ``STATE_NAMES``: the token caches, and what ``router_cache_prefill`` leaves of
    both router streams.  ``slots = 0``: one layer's column order (``W = 384 + R``), caches ``[B, T, width]``;
    ``slots = S``: ``S`` slots of 384 columns, then the operand, slot caches ``[S, B, T, width]``."""
    if not sequence_state_in_one_launch(block_size):
        return _sequence_state_by_parts(packed, slots, relation_dim, block_size, anchor_conv_weight, partner_conv_weight)
    return dict(zip(STATE_NAMES, _sequence_state(packed, slots, relation_dim, block_size, anchor_conv_weight,
                                                 partner_conv_weight)))


# Positions of the largest block whose router rows, with two rows of history, and convolved rows the kernel can hold in
# shared memory: (2 n + 2) rows of 256 bytes in 226 KB.  Longer blocks are copied and walked in device memory.
_STATE_BLOCK = 451


def sequence_state_in_one_launch(block_size: int) -> bool:
    return block_size <= _STATE_BLOCK


def _sequence_state_by_parts(packed: Tensor, slots: int, relation_dim: int, block_size: int, anchor_conv_weight: Tensor,
                             partner_conv_weight: Tensor) -> dict[str, Tensor]:
    (batch, length, width), n = packed.shape, max(slots, 1)
    if packed.dtype not in (torch.bfloat16, torch.float16) or slots < 0 or length % block_size != 0 \
            or width != 384 * n + relation_dim or anchor_conv_weight.numel() != 192 * n \
            or partner_conv_weight.numel() != 192 * n:
        raise ValueError("packed must be 16-bit [B, T, 384 * slots + R] of whole blocks and the conv weights [slots, 64, 3]")
    operand_at, anchor_at = (384 * n, 128) if slots else (128, 128 + relation_dim)

    def columns(at: int, size: int) -> Tensor:
        if not slots:
            return packed[..., at:at + size].contiguous()
        return torch.stack([packed[..., 384 * s + at:384 * s + at + size] for s in range(n)])

    state = {"anchor_keys": columns(0, 64), "partner_keys": columns(64, 64),
             "operand_cache": packed[..., operand_at:operand_at + relation_dim].contiguous(),
             "partner_anchor_cache": columns(anchor_at, 128)}
    for name in STATE_NAMES[4:]:
        tail = (length, 64) if name.endswith("cache") else (length // block_size, 4, 16)
        state[name] = packed.new_zeros((n, batch, *tail))
    weights = anchor_conv_weight.view(n, 64, 3), partner_conv_weight.view(n, 64, 3)
    for s in range(n):
        router = packed[..., 384 * s + anchor_at + 128:384 * s + anchor_at + 256]
        router_cache_prefill(router[..., :64], router[..., 64:], *[state[name][s] for name in STATE_NAMES[4:]],
                             weights[0][s], weights[1][s], block_size)
    return {name: t if slots or name in STATE_NAMES[:4] else t[0] for name, t in state.items()}


@torch.library.register_fake("relation_lm::sequence_state")
def _(packed, slots, relation_dim, block_size, anchor_conv_weight, partner_conv_weight):
    batch, length, lead = packed.size(0), packed.size(1), (slots,) if slots > 0 else ()
    wide = [packed.new_empty((*lead, batch, length, w)) for w in (64, 64, 128, 64, 64, 64, 64)]
    stats = [packed.new_empty((*lead, batch, length // block_size, 4, 16)) for _ in range(4)]
    return [wide[0], wide[1], packed.new_empty((batch, length, relation_dim)), *wide[2:], *stats]


@torch.library.custom_op("relation_lm::packed_projection_append", mutates_args=_APPEND_MUTATED, device_types="cuda")
def packed_projection_append(
    x: Tensor,
    weight: Tensor,
    anchor_keys: Tensor,
    partner_keys: Tensor,
    operand_cache: Tensor,
    partner_anchor_cache: Tensor,
    anchor_raw_cache: Tensor,
    partner_raw_cache: Tensor,
    anchor_conv_cache: Tensor,
    partner_conv_cache: Tensor,
    anchor_mean: Tensor,
    anchor_std: Tensor,
    partner_mean: Tensor,
    partner_std: Tensor,
    anchor_conv_weight: Tensor,
    partner_conv_weight: Tensor,
    position: Tensor,
    block_size: int,
) -> Tensor:
    """The packed projection of one decode position for all layers with ``sparse_cache_append`` in its
    epilogue (extension; decode batches of at most 16 rows, ``d`` 256 or 512): one launch writes the
    token-cache rows and updates both router streams of every layer, each output element by the
    thread that computed it.  Returns the packed rows ``[B, layers * (384 + R)]``; the state equals
    ``sparse_cache_append(skinny_projection(x, weight), ...)`` bit for bit."""
    device = _abi.require_cuda_contiguous(
        weight=weight, anchor_keys=anchor_keys, partner_keys=partner_keys, operand_cache=operand_cache,
        partner_anchor_cache=partner_anchor_cache, anchor_raw_cache=anchor_raw_cache,
        partner_raw_cache=partner_raw_cache, anchor_conv_cache=anchor_conv_cache,
        partner_conv_cache=partner_conv_cache, anchor_mean=anchor_mean, anchor_std=anchor_std,
        partner_mean=partner_mean, partner_std=partner_std, anchor_conv_weight=anchor_conv_weight,
        partner_conv_weight=partner_conv_weight)
    _abi.require_cuda_rows(x=x)
    _abi.require_position(position, device)
    layers, batch, max_t, rdim = operand_cache.shape
    width = 384 + rdim
    if x.shape[0] != batch or weight.shape != (layers * width, x.shape[1]) or anchor_keys.shape != (layers, batch, max_t, 64) \
            or partner_anchor_cache.shape != (layers, batch, max_t, 128) or anchor_raw_cache.shape != (layers, batch, max_t, 64) \
            or anchor_mean.size(0) != layers or anchor_conv_weight.shape != (layers, 64, 3):
        raise ValueError("caches must be [layers, B, T, width], weight [layers * (384 + R), d], conv weights [layers, 64, 3]")
    if anchor_conv_weight.dtype != torch.float32 or partner_conv_weight.dtype != torch.float32:
        raise ValueError("conv weights must be float32")
    dtype = _abi.same_dtype("16-bit operand", x, weight, anchor_keys, partner_keys, operand_cache, partner_anchor_cache,
                            anchor_raw_cache, partner_raw_cache, anchor_conv_cache, partner_conv_cache, anchor_mean,
                            anchor_std, partner_mean, partner_std)
    packed = torch.empty((batch, layers * width), device=device, dtype=x.dtype)
    with _abi.device_guard(device):
        _abi.check(_abi.LIB.rlm_packed_projection_append(
            _abi.ptr(x), x.stride(0), _abi.ptr(weight), _abi.ptr(packed), rdim, _abi.ptr(anchor_keys),
            _abi.ptr(partner_keys), _abi.ptr(operand_cache), _abi.ptr(partner_anchor_cache),
            _abi.ptr(anchor_raw_cache), _abi.ptr(partner_raw_cache), _abi.ptr(anchor_conv_cache),
            _abi.ptr(partner_conv_cache), _abi.ptr(anchor_mean), _abi.ptr(anchor_std), _abi.ptr(partner_mean),
            _abi.ptr(partner_std), _abi.ptr(anchor_conv_weight), _abi.ptr(partner_conv_weight), _abi.ptr(position),
            layers, batch, x.size(1), max_t, anchor_mean.size(2), int(block_size), dtype,
            _abi.ptr(_abi.status_tensor(device)), _abi.stream_ptr(device)))
    return packed


@packed_projection_append.register_fake
def _(x, weight, anchor_keys, partner_keys, operand_cache, partner_anchor_cache, anchor_raw_cache,
      partner_raw_cache, anchor_conv_cache, partner_conv_cache, anchor_mean, anchor_std, partner_mean,
      partner_std, anchor_conv_weight, partner_conv_weight, position, block_size):
    return x.new_empty((x.size(0), weight.size(0)))


def state_slide(tensors: list[Tensor], shifts: list[int], row_dim: int | list[int] = -2) -> None:
    """Slide position-indexed caches in place (extension; ``rlm_state_slide``): tensor ``k`` — contiguous,
    rows along ``row_dim`` (one value, or one per tensor: the position axis -2 of a cache ``[..., T, width]``,
    the block axis -3 of the router statistics ``[..., blocks, heads, width]``) — moves rows ``[shifts[k], rows)`` to the front and keeps its last
    ``shifts[k]`` rows as they were.  Up to 16 tensors per launch; longer lists take several launches.
    Not a registered operator: a decoder calls it between steps, outside its captured graph."""
    import ctypes

    if len(tensors) != len(shifts):
        raise ValueError("one shift per tensor")
    if not tensors:
        return
    device = tensors[0].device
    entries = []
    dims = list(row_dim) if isinstance(row_dim, (list, tuple)) else [row_dim] * len(tensors)
    if len(dims) != len(tensors):
        raise ValueError("one row_dim per tensor")
    for t, shift, axis in zip(tensors, shifts, dims):
        if t.numel() == 0:
            continue
        if not t.is_cuda or t.device != device or not t.is_contiguous():
            raise ValueError("state_slide takes contiguous CUDA tensors of one device")
        dim = int(axis) % t.dim()
        rows = t.size(dim)
        outer = 1
        for d in range(dim):
            outer *= t.size(d)
        inner = t.element_size()
        for d in range(dim + 1, t.dim()):
            inner *= t.size(d)
        if not 0 <= int(shift) < rows:
            raise ValueError("shift must be in [0, rows)")
        entries.append((t.data_ptr(), outer, rows, inner, int(shift)))
    for first in range(0, len(entries), 16):
        part = entries[first:first + 16]
        n = len(part)
        ptrs = (ctypes.c_void_p * n)(*[e[0] for e in part])
        cols = [(ctypes.c_int64 * n)(*[e[i] for e in part]) for i in (1, 2, 3, 4)]
        with _abi.device_guard(device):
            _abi.check(_abi.LIB.rlm_state_slide(ptrs, *cols, n, _abi.stream_ptr(device)))
