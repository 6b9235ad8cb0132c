"""``relation_lm::packed_projection`` — the packed sparse-cache projection on the tensor cores.

``out = x @ weight.T`` for bfloat16 / float16 operands: a hand-written sm_100a kernel
(TMA tile loads, ``tcgen05.mma`` with the accumulator in tensor memory).  It stands where the
reference project calls ``F.linear`` in ``PackedSparseCacheProjection.project``
(src/relation_lm/inference/packed_cache.py:52-57) and also serves the query-side router
projections.
"""
from __future__ import annotations

import torch
from torch import Tensor

from relation_lm.kernels import _abi

# The operators themselves are registered by csrc/torch_ops.cpp; the functions below document them.
_packed_projection = _abi.operator("packed_projection")
_layer_norm_cast = _abi.operator("layer_norm_cast")
_decode_embed_norm = _abi.operator("decode_embed_norm")
_decode_front = _abi.operator("decode_front")
_greedy_token = _abi.operator("greedy_token")
_few_rows_projection = _abi.operator("few_rows_projection")
_few_rows_projection_pair = _abi.operator("few_rows_projection_pair")
_skinny_projection = _abi.operator("skinny_projection")
_skinny_projection_greedy = _abi.operator("skinny_projection_greedy")
_skinny_projection_greedy_into = _abi.operator("skinny_projection_greedy_into")

_FUSED_NORM_ROWS = 16    # beyond this many rows normalising once beats normalising in every column tile


def packed_projection(x: Tensor, weight: Tensor, bias: Tensor | None = None) -> Tensor:
    """``x [rows, d] @ weight [n, d].T (+ bias [n])`` → ``[rows, n]`` in the operands' dtype (fp32
    accumulate; the optional fp32 bias is added before the result is rounded)."""
    return _packed_projection(x, weight, bias)


@torch.library.register_fake("relation_lm::packed_projection")
def _(x, weight, bias=None):
    return x.new_empty((x.size(0), weight.size(0)))


@torch.library.custom_op("relation_lm::packed_projection_slices", mutates_args=(), device_types="cuda")
def packed_projection_slices(x: Tensor, weight: Tensor, splits: int) -> Tensor:
    """Split-K form for few rows and a long reduction: ``splits`` CTAs share an output tile and the
    result comes back as fp32 slices ``[splits, rows, n]`` whose sum is ``x @ weight.T`` (the consumer,
    ``relation_norm_reduce_residual_norm_slices``, adds them up).  ``splits`` divides ``d / 64``."""
    device = _abi.require_cuda_rows(x=x)
    _abi.require_cuda_contiguous(weight=weight)
    if weight.device != device or weight.dim() != 2 or weight.size(1) != x.size(1):
        raise ValueError("weight must be [n_out, d_in] on the device of x")
    if x.dtype != weight.dtype or x.dtype not in (torch.bfloat16, torch.float16):
        raise ValueError("packed_projection takes bfloat16 or float16 operands of one dtype")
    rows, d_in = x.shape
    n_out = weight.size(0)
    out = torch.empty((int(splits), rows, n_out), device=device, dtype=torch.float32)
    with _abi.device_guard(device):
        _abi.check(_abi.LIB.rlm_packed_projection(
            _abi.ptr(x), x.stride(0), _abi.ptr(weight), None, _abi.ptr(out), rows, d_in, n_out,
            _abi.code(x), _abi.code(out), int(splits), _abi.ptr(_abi.status_tensor(device)),
            _abi.stream_ptr(device)))
    return out


@packed_projection_slices.register_fake
def _(x, weight, splits):
    return x.new_empty((splits, x.size(0), weight.size(0)), dtype=torch.float32)


def layer_norm_cast(x: Tensor, norm_weight: Tensor, norm_bias: Tensor, norm_eps: float, out: Tensor) -> None:
    """``out = layer_norm(x)`` for fp32 rows ``[rows, d]``, in the dtype of ``out``."""
    _layer_norm_cast(x, norm_weight, norm_bias, norm_eps, out)


@torch.library.register_fake("relation_lm::layer_norm_cast")
def _(x, norm_weight, norm_bias, norm_eps, out):
    return None


@torch.library.custom_op("relation_lm::norm_projection", mutates_args=(), device_types="cuda")
def norm_projection(x: Tensor, norm_weight: Tensor, norm_bias: Tensor, weight: Tensor,
                    norm_eps: float) -> Tensor:
    """``layer_norm(x) @ weight.T`` in one launch for fp32 rows: the rows are normalised in
    fp32, rounded to the weight dtype and multiplied on the tensor cores."""
    device = _abi.require_cuda_rows(x=x)
    _abi.require_cuda_contiguous(norm_weight=norm_weight, norm_bias=norm_bias, weight=weight)
    if x.dtype != torch.float32 or norm_weight.dtype != torch.float32 or norm_bias.dtype != torch.float32:
        raise ValueError("norm_projection takes fp32 rows and fp32 LayerNorm parameters")
    if weight.dim() != 2 or weight.size(1) != x.size(1) or norm_weight.numel() != x.size(1):
        raise ValueError("weight must be [n_out, d_in] and the norm parameters [d_in]")
    rows, d_in = x.shape
    if rows > _FUSED_NORM_ROWS:
        # normalise once into a 16-bit matrix, then the TMA-fed GEMM
        normalized = torch.empty((rows, d_in), device=device, dtype=weight.dtype)
        layer_norm_cast(x, norm_weight, norm_bias, norm_eps, normalized)
        return packed_projection(normalized, weight)
    out = torch.empty((rows, weight.size(0)), device=device, dtype=weight.dtype)
    with _abi.device_guard(device):
        _abi.check(_abi.LIB.rlm_norm_projection(
            _abi.ptr(x), x.stride(0), _abi.ptr(norm_weight), _abi.ptr(norm_bias), float(norm_eps),
            _abi.ptr(weight), _abi.ptr(out), rows, d_in, weight.size(0), _abi.code(weight),
            _abi.code(out), _abi.ptr(_abi.status_tensor(device)), _abi.stream_ptr(device)))
    return out


@norm_projection.register_fake
def _(x, norm_weight, norm_bias, weight, norm_eps):
    return x.new_empty((x.size(0), weight.size(0)), dtype=weight.dtype)


@torch.library.custom_op("relation_lm::decode_embed", mutates_args=(), device_types="cuda")
def decode_embed(tokens: Tensor, boundaries: Tensor, token_table: Tensor, boundary_table: Tensor,
                 position_table: Tensor, position: Tensor, scale: float) -> Tensor:
    """``(token_table[tokens] + boundary_table[boundaries]) * scale + position_table[position]``
    for one decode position, ``[B, d]`` fp32."""
    device = _abi.require_cuda_contiguous(tokens=tokens, boundaries=boundaries,
                                          token_table=token_table, boundary_table=boundary_table,
                                          position_table=position_table)
    _abi.require_position(position, device)
    if tokens.dtype != torch.int64 or boundaries.dtype != torch.int64 or position_table.dtype != torch.float32:
        raise ValueError("ids must be int64 and the position table float32")
    batch, d_model = tokens.numel(), token_table.size(1)
    out = torch.empty((batch, d_model), device=device, dtype=torch.float32)
    with _abi.device_guard(device):
        _abi.check(_abi.LIB.rlm_decode_embed(
            _abi.ptr(tokens), _abi.ptr(boundaries), _abi.ptr(token_table), _abi.ptr(boundary_table),
            _abi.ptr(position_table), _abi.ptr(position), float(scale), _abi.ptr(out), batch, d_model,
            token_table.size(0), boundary_table.size(0), position_table.size(0),
            _abi.same_dtype("embedding table", token_table, boundary_table),
            None, None, None, None, None, None, 0.0, 0,
            _abi.ptr(_abi.status_tensor(device)), _abi.stream_ptr(device)))
    return out


@decode_embed.register_fake
def _(tokens, boundaries, token_table, boundary_table, position_table, position, scale):
    return token_table.new_empty((tokens.numel(), token_table.size(1)), dtype=torch.float32)


def decode_embed_norm(tokens: Tensor, boundaries: Tensor, token_table: Tensor, boundary_table: Tensor,
                      position_table: Tensor, position: Tensor, scale: float, norm1_weight: Tensor,
                      norm1_bias: Tensor, normalized1: Tensor, norm2_weight: Tensor, norm2_bias: Tensor,
                      normalized2: Tensor, norm_eps: float) -> Tensor:
    """``decode_embed`` that also writes two LayerNorms of the embedded rows in the outputs' dtype
    (``normalized1`` with the memory norm for the packed projection, ``normalized2`` with the first
    layer's input norm for its query projection); returns the fp32 rows."""
    return _decode_embed_norm(tokens, boundaries, token_table, boundary_table, position_table, position, scale,
                              norm1_weight, norm1_bias, normalized1, norm2_weight, norm2_bias, normalized2, norm_eps)


@torch.library.register_fake("relation_lm::decode_embed_norm")
def _(tokens, boundaries, token_table, boundary_table, position_table, position, scale, norm1_weight,
      norm1_bias, normalized1, norm2_weight, norm2_bias, normalized2, norm_eps):
    return token_table.new_empty((tokens.numel(), token_table.size(1)), dtype=torch.float32)


def l2_prefetch(tensors: list[Tensor]) -> None:
    """Issue L2 prefetches for up to 16 CUDA tensors (their storage from the first element to the last), in
    order, on the current stream (extension; see ``rlm_l2_prefetch``).  Not a registered operator: it has no
    outputs and no effect on values."""
    import ctypes

    tensors = [t for t in tensors if t is not None and t.numel() > 0]
    if not tensors:
        return
    if len(tensors) > 16:
        raise ValueError("at most 16 tensors per call")
    device = tensors[0].device
    for t in tensors:
        if not t.is_cuda or t.device != device or not t.is_contiguous():
            raise ValueError("l2_prefetch takes contiguous CUDA tensors of one device")
    ranges = (ctypes.c_void_p * len(tensors))(*[t.data_ptr() for t in tensors])
    sizes = (ctypes.c_int64 * len(tensors))(*[t.numel() * t.element_size() for t in tensors])
    with _abi.device_guard(device):
        _abi.check(_abi.LIB.rlm_l2_prefetch(ranges, sizes, len(tensors), _abi.stream_ptr(device)))


def decode_front_supported(batch: int, d_model: int, n_first: int, dtype: torch.dtype) -> bool:
    return batch <= 16 and d_model in (256, 512) and n_first % 8 == 0 and dtype in (torch.bfloat16, torch.float16)


def decode_front(tokens: Tensor, boundaries: Tensor, token_table: Tensor, boundary_table: Tensor,
                 position_table: Tensor, position: Tensor, scale: float, norm1_weight: Tensor, norm1_bias: Tensor,
                 norm2_weight: Tensor, norm2_bias: Tensor, norm_eps: float, weight: Tensor, n_first: int,
                 norm1_out: Tensor, norm2_out: Tensor, out_second: Tensor) -> tuple[Tensor, Tensor]:
    """The front of a decode step in one launch (extension): embedding of one position, two LayerNorms
    of the embedded rows and one projection of each — ``weight[:n_first]`` of the ``norm1`` rows (returned,
    ``[B, n_first]``) and ``weight[n_first:]`` of the ``norm2`` rows (into ``out_second``).  Also returns
    the embedded rows (fp32) and stores the two normalised copies.  At most 16 rows, ``d`` 256 or 512."""
    return _decode_front(tokens, boundaries, token_table, boundary_table, position_table, position, scale,
                         norm1_weight, norm1_bias, norm2_weight, norm2_bias, norm_eps, weight, n_first, norm1_out,
                         norm2_out, out_second)


@torch.library.register_fake("relation_lm::decode_front")
def _(tokens, boundaries, token_table, boundary_table, position_table, position, scale, norm1_weight, norm1_bias,
      norm2_weight, norm2_bias, norm_eps, weight, n_first, norm1_out, norm2_out, out_second):
    batch = tokens.numel()
    return (token_table.new_empty((batch, token_table.size(1)), dtype=torch.float32),
            weight.new_empty((batch, n_first)))


def greedy_token(logits: Tensor, vocab: int, position: Tensor | None = None) -> Tensor:
    """``logits[:, :vocab].argmax(-1)`` (ties to the lowest index) as int64 ``[rows]``; with
    ``position`` (a 0-d int64 device tensor) the position is advanced by one in the same launch."""
    return _greedy_token(logits, vocab, position)




@torch.library.register_fake("relation_lm::greedy_token")
def _(logits, vocab, position):
    return logits.new_empty((logits.size(0),), dtype=torch.int64)


def few_rows_projection_supported(rows: int, d_in: int, dtype: torch.dtype) -> bool:
    """Whether ``few_rows_projection`` takes these sizes."""
    return 1 <= rows <= 64 and d_in % 4 == 0 and dtype == torch.float32


def few_rows_projection(out: Tensor, x: Tensor, weight: Tensor, bias: Tensor | None = None) -> None:
    """``out = x [rows <= 64, d] @ weight [n, d].T (+ bias)`` in single precision (extension): the products of one
    decode position, streams of their weight matrices."""
    _few_rows_projection(out, x, weight, bias)


@torch.library.register_fake("relation_lm::few_rows_projection")
def _(out, x, weight, bias=None):
    return None


def few_rows_projection_pair(out: Tensor, out2: Tensor, x: Tensor, weight: Tensor, weight2: Tensor,
                             bias2: Tensor | None = None) -> None:
    """``few_rows_projection`` with two weights for the same rows in one launch: ``out = x @ weight.T``,
    ``out2 = x @ weight2.T (+ bias2)``."""
    _few_rows_projection_pair(out, out2, x, weight, weight2, bias2)


@torch.library.register_fake("relation_lm::few_rows_projection_pair")
def _(out, out2, x, weight, weight2, bias2=None):
    return None


def skinny_projection_supported(rows: int, d_in: int, dtype: torch.dtype) -> bool:
    """Whether ``skinny_projection`` serves these sizes (a handful of rows, a weight row in registers)."""
    return 1 <= rows <= 16 and d_in in (256, 512) and dtype in (torch.bfloat16, torch.float16)


def skinny_projection(x: Tensor, weight: Tensor, bias: Tensor | None = None) -> Tensor:
    """``x [rows <= 16, d] @ weight [n, d].T (+ bias)`` on the CUDA cores (extension): for a decode
    batch the product is a stream of the weight matrix, read once by whole warps with no tensor-memory
    or tensor-map set-up.  Same contract as ``packed_projection``; ``d`` must be 256 or 512."""
    return _skinny_projection(x, weight, bias)


@torch.library.register_fake("relation_lm::skinny_projection")
def _(x, weight, bias=None):
    return x.new_empty((x.size(0), weight.size(0)))


def skinny_projection_greedy(x: Tensor, weight: Tensor, bias: Tensor | None, vocab: int, scratch: Tensor,
                             position: Tensor | None) -> tuple[Tensor, Tensor]:
    """The output head of a greedy decode step in one launch (extension): ``logits = x @ weight.T + bias``
    and ``next_token = logits[:, :vocab].argmax(-1)`` (lowest index on ties; int64), and with ``position``
    the device position advanced by one.  ``scratch``: a zeroed uint8 tensor of
    ``skinny_argmax_scratch_bytes()`` bytes, allocated once by the caller and left zero by every launch."""
    return _skinny_projection_greedy(x, weight, bias, vocab, scratch, position)


@torch.library.register_fake("relation_lm::skinny_projection_greedy")
def _(x, weight, bias, vocab, scratch, position):
    return x.new_empty((x.size(0), weight.size(0))), x.new_empty((x.size(0),), dtype=torch.int64)


def skinny_projection_greedy_into(x: Tensor, weight: Tensor, bias: Tensor | None, vocab: int, scratch: Tensor,
                                  position: Tensor | None, next_token: Tensor) -> Tensor:
    """``skinny_projection_greedy`` writing the chosen tokens into the caller's ``next_token`` ``[rows]``
    (int64) — which may be a device view of pinned host memory (``mapped_host_view``): the choice then
    reaches the host without a copy of its own.  Returns the logits."""
    return _skinny_projection_greedy_into(x, weight, bias, vocab, scratch, position, next_token)


@torch.library.register_fake("relation_lm::skinny_projection_greedy_into")
def _(x, weight, bias, vocab, scratch, position, next_token):
    return x.new_empty((x.size(0), weight.size(0)))


class _MappedHost:
    """Pinned host memory presented through ``__cuda_array_interface__`` (with unified addressing the
    device address of pinned memory is its host address)."""

    def __init__(self, host: Tensor) -> None:
        code = {torch.int64: "<i8", torch.int32: "<i4", torch.float32: "<f4", torch.uint8: "|u1"}[host.dtype]
        self.__cuda_array_interface__ = {"shape": tuple(host.shape), "typestr": code,
                                         "data": (host.data_ptr(), False), "version": 2}
        self.host = host


def mapped_host_view(host: Tensor, device: torch.device) -> Tensor:
    """A CUDA tensor over the pinned, contiguous host tensor ``host``: kernels that take it read or write
    the host memory directly (a few bytes of ids in, a few bytes of choices out: cheaper than a copy node
    per transfer in a decode graph).  The host sees a kernel's writes once the stream is synchronised.  The
    view keeps ``host`` alive."""
    if host.is_cuda or not host.is_pinned() or not host.is_contiguous():
        raise ValueError("mapped_host_view takes a pinned, contiguous host tensor")
    holder = _MappedHost(host)
    view = torch.as_tensor(holder, device=device)
    if view.data_ptr() != host.data_ptr() or not view.is_cuda:
        raise RuntimeError("the device view does not alias the host tensor")
    view._mapped_host = holder
    return view


def skinny_argmax_scratch_bytes() -> int:
    return int(_abi.LIB.rlm_skinny_argmax_scratch_bytes())
