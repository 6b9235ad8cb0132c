"""Stateful sparse decode: one new position per call, all history in caches.

The step is the composition the reference's decode operators were written for (its own
driver is not public; the order follows docs/architecture.md:26-40 and
docs/benchmarks.md:87-113 of the reference project):

1. embed the new token, ``memory = LayerNorm(x)``; one packed projection of ``memory`` for
   every layer (packed_cache.py:52-57) followed by ``sparse_cache_append`` (token-cache rows
   + ``router_cache_update`` of all layers, one launch);
2. per layer: ``LayerNorm(hidden)`` -> one 256-wide query-side projection ->
   ``relation_select_packed`` -> ``relation_hidden_cache_update_out`` -> second relation-MLP layer
   -> ``relation_norm_reduce`` -> ``hidden += sigmoid(mix) * context``;
3. final LayerNorm, tied token head, boundary head.

Every state tensor is allocated once and mutated in place; ``position`` lives on the device
and is advanced there, so a captured CUDA graph of ``step`` replays for successive positions.
"""
from __future__ import annotations

from types import SimpleNamespace

import torch
import torch.nn.functional as F
from torch import Tensor

from relation_lm.inference.routed_model import RoutedRelationLM
from relation_lm.kernels import _abi
from relation_lm.kernels.packed_projection import (decode_embed_norm, decode_front, decode_front_supported,
                                                    few_rows_projection, few_rows_projection_pair,
                                                    few_rows_projection_supported,
                                                    greedy_token, l2_prefetch, layer_norm_cast,
                                                    mapped_host_view, packed_projection, packed_projection_slices,
                                                    skinny_argmax_scratch_bytes, skinny_projection,
                                                    skinny_projection_greedy, skinny_projection_greedy_into,
                                                    skinny_projection_supported)
from relation_lm.kernels.relation_reduce import (expanded_cache_append, expanded_cache_append_packed,
                                                 relation_layer_tail, relation_layer_tail_supported,
                                                 relation_layer_tail_wide, relation_layer_tail_wide_supported,
                                                 relation_hidden_cached_out,
                                                 relation_hidden_cache_update_out,
                                                 relation_norm_reduce_residual_norm,
                                                 relation_norm_reduce_residual_norm_project,
                                                 relation_norm_reduce_residual_norm_slices,
                                                 relation_norm_reduce, relation_tail)
from relation_lm.kernels.relation_select import relation_select_packed
from relation_lm.kernels.relation_layer import relation_layer, relation_layer_supported
from relation_lm.kernels.router_cache import packed_projection_append, sparse_cache_append, state_slide


class StatefulDecoder:
    def __init__(self, model: RoutedRelationLM, batch: int, device="cuda",
                 dtype: torch.dtype = torch.bfloat16, fused_tail: bool = False,
                 programmatic_launch: bool = True, second_layer_split: bool = False,
                 fused_query: bool | None = None, layer_tail: bool | None = None,
                 skinny: bool | None = None, append_in_projection: bool | None = None,
                 whole_layer: bool | None = None, fused_front: bool | None = None,
                 prefetch: bool | None = None) -> None:
        cfg = model.config
        self.programmatic_launch = bool(programmatic_launch)
        self.config, self.batch, self.device, self.dtype = cfg, int(batch), torch.device(device), dtype
        self.w = model.decode_weights(self.device, dtype)
        self.input_scale = float(model.input_scale)
        L, B, T, R, H = cfg.layers, self.batch, cfg.max_context, cfg.relation_dim, cfg.hidden_dim
        nb = T // cfg.block_size

        def zeros(*shape, dt=dtype):
            return torch.zeros(*shape, device=self.device, dtype=dt)

        self.anchor_keys = zeros(L, B, T, 64)
        self.partner_keys = zeros(L, B, T, 64)
        self.operand_cache = zeros(L, B, T, R)
        self.partner_anchor_cache = zeros(L, B, T, 128)
        self.expanded_cache = zeros(L, B, T, 2 * H)
        self.router_caches = [zeros(L, B, T, 64) for _ in range(4)]   # raw a, raw p, conv a, conv p
        self.router_stats = [zeros(L, B, nb, 4, 16) for _ in range(4)]  # mean a, std a, mean p, std p
        self.position = torch.zeros((), device=self.device, dtype=torch.int64)
        self.last_selection: list[tuple[Tensor, Tensor]] = []
        # When set to a list, the fused step appends one dict of cloned intermediates per layer
        # (and one for the embedding / append stage), so that a checker can feed every kernel's own
        # inputs to an independent implementation.  Not for captured graphs.
        self.trace: list[dict[str, Tensor]] | None = None
        self.last_final: Tensor | None = None           # final LayerNorm output of the last step
        self._graph = None
        # Low-precision decode batches take the fused path: LayerNorm folded into the tcgen05
        # projections, 16-bit relation hidden states, residual update inside norm-reduce.
        self.fused = (dtype in (torch.bfloat16, torch.float16)
                      and cfg.d_model % 64 == 0 and cfg.d_model <= 1024)
        # The single-launch tail (second MLP layer + norm-reduce + residual) is optional: at
        # decode batch sizes its one-CTA finalisation costs more than the launch it saves.
        self.fused_tail = fused_tail and self.fused and 128 % cfg.k_max == 0 and cfg.k_max <= 32
        # One tensor-core launch expands the position's operand rows of all layers (shapes permitting).
        self.stacked_expand = self.fused and R % 64 == 0 and H % 128 == 0
        # Second relation-MLP layer: cuBLAS (F.linear) by default.  Optionally, with at most one row
        # tile (B * K <= 128), the library's GEMM splits the reduction over the hidden width across
        # several CTAs and norm-reduce sums the slices: no library call in the step, a few percent slower.
        self.second_layer_splits = 1
        if self.fused and second_layer_split and B * cfg.k_max <= 128 and H % 64 == 0 and cfg.d_model % 32 == 0:
            blocks = H // 64
            self.second_layer_splits = next((s for s in (4, 2) if blocks % s == 0 and blocks // s >= 2), 1)
        if self.second_layer_splits > 1:
            self.b2_f32 = self.w["b2"].float().contiguous()                    # [L, d], dtype of the norm parameters
        # Next layer's query projection inside norm-reduce (a cluster of CTAs per row): one launch
        # fewer per layer for batches of a few rows; larger batches keep the tensor-core projection
        # (12 layers of d 768, us per step with / without: 364 / 376 for 12 rows, 467 / 427 for 16,
        # whose clusters no longer all find room at once).
        n_query = self.w["w_query"].shape[1]
        can_fuse_query = (self.fused and not self.fused_tail and self.second_layer_splits == 1
                          and n_query % 32 == 0 and n_query <= 256)
        self.fused_query = can_fuse_query and (B <= 12 if fused_query is None else bool(fused_query))
        # The whole relation tail of a layer (relation hidden, second MLP layer, norm-reduce, residual,
        # next LayerNorm, next query projection) as ONE cluster launch with the hidden states on chip:
        # two launches per layer and no library GEMM in the step, for small batches of d <= 512 and of d 768.
        sizes = (B, cfg.k_max, R, H, cfg.d_model, n_query, dtype)
        wide = cfg.d_model == 768
        can_tail = (self.fused and not self.fused_tail and self.second_layer_splits == 1 and self.stacked_expand and B <= 64
                    and (relation_layer_tail_wide_supported(*sizes) if wide else relation_layer_tail_supported(*sizes)))
        self._tail = relation_layer_tail_wide if wide else relation_layer_tail
        # (d 768 below 256 pairs; us per step of 12 layers, context 1024, with the tail / with four or five launches a layer:
        # 250 / 303 for one sequence, 269 / 341 for 8, 400 / 483 for 28; 397 / 355 for 32 at context 512, whose hidden states
        # take the tensor-core kernel.  From 57 sequences on, K <= 4, its eight clusters of 16 CTAs take two waves, as seven
        # run at a time, and it is still the faster: 373 / 622 for 56 of K 4, 537 / 653 for 57, 623 / 652 for 63, 616 / 653
        # for 64 of K 3, 516 / 634 of K 1)
        by_default = can_tail and not (wide and B * cfg.k_max >= 256)
        self.layer_tail = by_default if layer_tail is None else (bool(layer_tail) and can_tail)
        if self.layer_tail:
            self.fused_query = False
        self.query = zeros(B, n_query) if self.fused else zeros(L, B, n_query)
        # ... and the selector can run in front of the tail inside the same cluster: one launch per layer.
        # Off by default: with the step's working set cold in L2 it measured 3-5 % slower than the two
        # launches (equal when warm), whose selector overlaps the tail's weight loads just as well.
        can_whole = self.layer_tail and relation_layer_supported(
            B, cfg.k_max, R, H, cfg.d_model, n_query, dtype, T, nb, self.w["anchor_bias"].shape[-1],
            cfg.local_window, cfg.top_blocks)
        self.whole_layer = bool(whole_layer) and can_whole
        # Projections of a handful of rows stream their weights through the CUDA cores (no tensor-memory
        # set-up); the head's launch then also takes the greedy arg-max and the position increment.
        can_skinny = self.fused and skinny_projection_supported(B, cfg.d_model, dtype)
        self.skinny = can_skinny if skinny is None else (bool(skinny) and can_skinny)
        # ... and the packed projection can take the cache append and router update into its epilogue
        # (one launch fewer; off by default: the channels' serial statistics in the epilogue cost more
        # than the separate, fully parallel append launch that overlaps its neighbours)
        self.append_in_projection = bool(append_in_projection) and self.skinny
        # ... and the step's front (embedding, two LayerNorms, packed projection, layer 0's query projection)
        # is one launch of the same kind over the two weight matrices stacked: three launches fewer
        can_front = (self.skinny and not self.append_in_projection and (self.fused_query or self.layer_tail)
                     and decode_front_supported(B, cfg.d_model, self.w["w_packed"].shape[0], dtype))
        self.fused_front = can_front if fused_front is None else (bool(fused_front) and can_front)
        if self.fused_front:
            self.front_weight = torch.cat((self.w["w_packed"], self.w["w_query"][0]), 0).contiguous()
        # A step of a small batch is a chain of dependent launches on a fraction of the SMs; when it
        # starts with a cold L2 every one of them first waits for its weights and caches to come from
        # DRAM.  One launch on a side stream at the head of the step can ask for all of them at once.
        # Off by default: measured 3-5 us SLOWER per step (cold and warm) than letting every kernel
        # fetch its own data under programmatic launch; the fork and join cost more than they hide.
        self.prefetch = bool(prefetch) and self.fused
        self._side_stream = torch.cuda.Stream(self.device) if self.prefetch else None
        self._project = skinny_projection if self.skinny else packed_projection
        if self.skinny:
            self.argmax_scratch = torch.zeros(skinny_argmax_scratch_bytes(), device=self.device, dtype=torch.uint8)
        self.relation_hidden = zeros(B, cfg.k_max, H)
        self.normalized = zeros(B, cfg.d_model)                 # LayerNorm'd input of the next projection
        self.memory_normalized = zeros(B, cfg.d_model)          # memory-norm'd input of the packed projection
        if not self.fused:
            # rows of whole 16-byte chunks up to 1024 wide: LayerNorms inside the kernels that make their input
            self.kernel_norms = cfg.d_model % 8 == 0 and cfg.d_model <= 1024
            # The products of a position's rows by the library's own kernel, and with it the whole step under
            # programmatic launch (libraries' kernels in between would wait for nothing that it lets run early).
            # From nine sequences on libraries have the better products (16 rows of the 16 256 heads at d 768: 36 us, 28).
            self.few_rows = (self.kernel_norms and B <= 8 and H % 4 == 0
                             and few_rows_projection_supported(B * cfg.k_max, cfg.d_model, dtype))
            if self.few_rows:
                self.packed_rows = zeros(B, self.w["w_packed"].shape[0])
                self.second_rows = zeros(B, cfg.k_max, cfg.d_model)
            # The heads too, unless their weights, which may be the model's own, start off a 16-byte boundary, or are so many
            # rows that libraries stream them faster (us, library / own kernel: one row of d 768, 16 256 columns 22.9 / 11.0,
            # 32 000 18.9 / 21.1, 128 256 61 / 71; eight rows 16 256 26.2 / 22.5, 32 000 42.8 / 43.2, 50 304 64 / 66, of d 1024
            # 128 256 169 / 212; two to four rows and d 256 are the kernel's at every size: four rows of d 768, 128 256 1.47 x).
            columns = cfg.vocab_size + cfg.boundary_vocab_size
            many = cfg.d_model > 256 and (columns > 24_000 if B == 1 else columns > 40_000 and B > 4)
            self.few_heads = self.few_rows and not many and all(self.w[n].data_ptr() % 16 == 0 for n in ("token_embedding", "boundary_w"))
            # one product for both heads where its column slices are dense matrices, as two products' results are
            if B == 1 and not self.few_heads:
                self.head_weight = torch.cat((self.w["token_embedding"], self.w["boundary_w"]), 0).contiguous()
                self.head_bias = torch.cat((zeros(cfg.vocab_size), self.w["boundary_b"]))
        else:
            self.head_weight = torch.cat((self.w["token_embedding"], self.w["boundary_w"]), 0).contiguous()
            pad = (-self.head_weight.size(0)) % 128        # whole 128-column tiles for the projection kernel
            if pad:
                self.head_weight = torch.cat((self.head_weight, zeros(pad, cfg.d_model)), 0).contiguous()
            # the boundary head's bias rides in the projection's epilogue (token columns: zero)
            self.head_bias = torch.zeros(self.head_weight.size(0), device=self.device, dtype=torch.float32)
            self.head_bias[cfg.vocab_size:cfg.vocab_size + cfg.boundary_vocab_size] = self.w["boundary_b"].float()

        self._layers = [self._layer_views(l) for l in range(L)]
        if not self.fused and self.few_rows:
            # what the grouped calls of the single-precision step take before and behind the position
            w = self.w
            self._front = ((w["token_embedding"], w["boundary_embedding"], w["position_embedding"]),
                           (self.input_scale, w["memory_norm_w"], w["memory_norm_b"], self.memory_normalized, w["input_norm_w"][0],
                            w["input_norm_b"][0], self.normalized, cfg.norm_eps, self.packed_rows, w["w_packed"], self.anchor_keys,
                            self.partner_keys, self.operand_cache, self.partner_anchor_cache, *self.router_caches,
                            *self.router_stats, w["anchor_conv_weight"], w["partner_conv_weight"], cfg.block_size))
            for layer in self._layers:
                layer.grouped = ((layer.w_query, layer.query, *layer.selection),
                                 (cfg.local_window, cfg.top_blocks, cfg.k_max, cfg.strict_valid, self.relation_hidden, *layer.caches,
                                  *layer.first_layer, self.second_rows, *layer.second_layer, *layer.relation_norm, cfg.norm_eps))

    # ------------------------------------------------------------------ state
    def reset(self) -> None:
        for t in (self.anchor_keys, self.partner_keys, self.operand_cache, self.partner_anchor_cache,
                  self.expanded_cache, *self.router_caches, *self.router_stats):
            t.zero_()
        self.position.zero_()

    def slide(self, blocks: int = 1) -> None:
        """Drop the oldest ``blocks`` router blocks of every sequence and lower the position by as
        many rows (``relation_lm.kernels.router_cache.state_slide``): how a decoder goes on once its
        position has reached ``max_context``.  Afterwards position ``p`` of the state is what position
        ``p + blocks * block_size`` was — keys, operands, expanded rows, router caches and the
        statistics of every block, none of them recomputed — so later steps choose among the rows a
        ring buffer of ``max_context`` rows would still hold, and count positions (the position
        embedding, the ``ceil(log2(t + 2))`` partner limit) from the oldest row kept.  One launch for
        the caches and statistics and one for the position, on the current stream, between steps
        (outside the captured graph, whose buffers it leaves where they are)."""
        cfg = self.config
        blocks = int(blocks)
        if not 0 < blocks < cfg.max_context // cfg.block_size:
            raise ValueError("slide by at least one block and fewer than the context holds")
        rows = blocks * cfg.block_size
        caches = [self.anchor_keys, self.partner_keys, self.operand_cache, self.partner_anchor_cache,
                  self.expanded_cache, *self.router_caches]
        state_slide(caches + list(self.router_stats), [rows] * len(caches) + [blocks] * 4,
                    row_dim=[-2] * len(caches) + [-3] * 4)
        self.position.sub_(rows)

    def state_bytes(self) -> int:
        tensors = (self.anchor_keys, self.partner_keys, self.operand_cache, self.partner_anchor_cache,
                   self.expanded_cache, *self.router_caches, *self.router_stats)
        return sum(t.numel() * t.element_size() for t in tensors)

    # ------------------------------------------------------------------ one position
    def step(self, tokens: Tensor, boundaries: Tensor, keep_selection: bool = False):
        """Consume one token per sequence at the current position; returns (token logits
        ``[B, V]``, boundary logits ``[B, Vb]``) and advances the position."""
        if self.fused:
            # The fused step keeps the selector's rule for programmatic launch: the caches are
            # written by the append, two launches before the first selector.
            previous = _abi.set_programmatic_launch(self.programmatic_launch)
            try:
                return self._step_fused(tokens, boundaries, keep_selection)
            finally:
                _abi.set_programmatic_launch(previous)
        if not self.few_rows or torch.compiler.is_compiling():      # (a tracer cannot follow the switch)
            return self._step_unfused(tokens, boundaries, keep_selection)
        previous = _abi.set_programmatic_launch(self.programmatic_launch)
        try:
            return self._step_unfused(tokens, boundaries, keep_selection)
        finally:
            _abi.set_programmatic_launch(previous)

    def step_greedy(self, tokens: Tensor, boundaries: Tensor, chosen_out: Tensor | None = None) -> Tensor:
        """One step followed by the greedy choice: returns the next token ids ``[B]`` (int64) and
        advances the position.  On the fused path the arg-max and the position increment are one
        launch of the library; with ``chosen_out`` (int64 ``[B]``, skinny fused path only) the choice is
        written there — a device view of pinned host memory included."""
        if chosen_out is not None and not (self.fused and self.skinny):
            raise ValueError("chosen_out needs the fused path with the head projection's greedy launch")
        if not self.fused:
            token_logits, _ = self.step(tokens, boundaries)
            return token_logits.argmax(-1)
        previous = _abi.set_programmatic_launch(self.programmatic_launch)
        try:
            if self.skinny:
                return self._step_fused(tokens, boundaries, False, advance=False, greedy=True, chosen_out=chosen_out)
            self._step_fused(tokens, boundaries, False, advance=False)
            return greedy_token(self.last_logits, self.config.vocab_size, self.position)
        finally:
            _abi.set_programmatic_launch(previous)

    def _step_unfused(self, tokens: Tensor, boundaries: Tensor, keep_selection: bool):
        """The step without the tensor-core projections (single precision, widths they do not take).  A step
        of one sequence is bound by the host, so what can ride in a kernel does: the embedding with both its
        LayerNorms, and norm-reduce with the residual update and the next LayerNorm."""
        cfg, w = self.config, self.w
        pos, K = self.position, cfg.k_max
        if self.kernel_norms:
            tokens, boundaries = self._ids(tokens, boundaries)
        # ... and its operators are called from native code, a call for a whole group of them, where nobody wants the
        # selections in between.
        grouped = self.few_rows and not keep_selection
        hidden = NotImplemented
        if grouped:
            hidden = _abi.direct_call("single_precision_front", tokens, boundaries, *self._front[0], pos, *self._front[1])
        if hidden is NotImplemented:
            hidden = self._front_unfused(tokens, boundaries)
        if keep_selection:
            self.last_selection = []
        for layer in self._layers:
            # the last layer's goes to a tensor of this step's own: it stays behind as `last_final`
            normalized = torch.empty_like(self.normalized) if layer is self._layers[-1] else self.normalized
            if grouped and _abi.direct_call("single_precision_layer", self.normalized, *layer.grouped[0], pos, *layer.grouped[1],
                                            hidden, layer.mix, *layer.next_norm, normalized) is not NotImplemented:
                continue
            if self.few_rows:
                few_rows_projection(layer.query, self.normalized, layer.w_query, None)        # [B, 256]
            else:
                torch.mm(self.normalized, layer.w_query_t, out=layer.query)
            anchor, _, partner, partner_score = relation_select_packed(
                *layer.selection, pos, cfg.local_window, cfg.top_blocks, K, cfg.strict_valid)
            relation_hidden_cache_update_out(self.relation_hidden, *layer.caches, anchor, partner, *layer.first_layer, pos)
            if self.few_rows:
                raw = self.second_rows                                                  # [B, K, d]
                few_rows_projection(raw.view(-1, cfg.d_model), self.relation_hidden.view(-1, cfg.hidden_dim), *layer.second_layer)
            else:
                raw = F.linear(self.relation_hidden, *layer.second_layer)
            if self.kernel_norms:
                relation_norm_reduce_residual_norm(raw, partner_score, *layer.relation_norm, pos, cfg.norm_eps, hidden,
                                                   layer.mix, *layer.next_norm, cfg.norm_eps, normalized)
            else:
                context = relation_norm_reduce(raw, partner_score, *layer.relation_norm, pos, cfg.norm_eps)
                torch.addcmul(hidden, context, layer.mix, out=hidden)
                self._normalize(hidden, *layer.next_norm, normalized)
            if keep_selection:
                self.last_selection.append((anchor, partner))
        self.last_final = normalized
        if grouped and self.few_heads:
            heads = _abi.direct_call("single_precision_heads", normalized, w["token_embedding"], w["boundary_w"], w["boundary_b"], pos)
            if heads is not NotImplemented:
                return heads
        if self.few_heads:
            heads = normalized.new_empty(self.batch, cfg.vocab_size), normalized.new_empty(self.batch, cfg.boundary_vocab_size)
            few_rows_projection_pair(*heads, normalized, w["token_embedding"], w["boundary_w"], w["boundary_b"])
        elif self.batch == 1:
            logits = F.linear(normalized, self.head_weight, self.head_bias)
            heads = logits[:, :cfg.vocab_size], logits[:, cfg.vocab_size:]
        else:
            heads = F.linear(normalized, w["token_embedding"]), F.linear(normalized, w["boundary_w"], w["boundary_b"])
        pos.add_(1)
        return heads

    def _front_unfused(self, tokens: Tensor, boundaries: Tensor) -> Tensor:
        """The embedded rows; their LayerNorms, packed projection and cache rows of the position on the way."""
        cfg, w, pos = self.config, self.w, self.position
        if self.kernel_norms:
            hidden = decode_embed_norm(tokens, boundaries, w["token_embedding"], w["boundary_embedding"],
                                       w["position_embedding"], pos, self.input_scale,
                                       w["memory_norm_w"], w["memory_norm_b"], self.memory_normalized,
                                       w["input_norm_w"][0], w["input_norm_b"][0], self.normalized, cfg.norm_eps)
        else:
            x = (F.embedding(tokens, w["token_embedding"]) + F.embedding(boundaries, w["boundary_embedding"])).float()
            hidden = x * self.input_scale + w["position_embedding"].index_select(0, pos.view(1))
            self._normalize(hidden, w["memory_norm_w"], w["memory_norm_b"], self.memory_normalized)
            self._normalize(hidden, w["input_norm_w"][0], w["input_norm_b"][0], self.normalized)
        if self.few_rows:
            packed = self.packed_rows                                 # [B, layers * 512]
            few_rows_projection(packed, self.memory_normalized, w["w_packed"], None)
        else:
            packed = F.linear(self.memory_normalized, w["w_packed"])
        sparse_cache_append(packed, self.anchor_keys, self.partner_keys, self.operand_cache,
                            self.partner_anchor_cache, *self.router_caches, *self.router_stats,
                            w["anchor_conv_weight"], w["partner_conv_weight"], pos, cfg.block_size)
        return hidden

    @staticmethod
    def _ids(tokens: Tensor, boundaries: Tensor) -> tuple[Tensor, Tensor]:
        """Ids as an embedding lookup takes them (32 bits, one for all sequences), as the kernel does: int64 ``[B]`` each."""
        if tokens.shape != boundaries.shape:
            tokens, boundaries = torch.broadcast_tensors(tokens, boundaries)
        if tokens.dim() != 1:
            if tokens.dim() > 1:
                raise ValueError("token and boundary ids must be [B]")
            tokens, boundaries = tokens.view(1), boundaries.view(1)
        if tokens.dtype == torch.int32:
            tokens = tokens.long()
        if boundaries.dtype == torch.int32:
            boundaries = boundaries.long()
        return tokens.contiguous(), boundaries.contiguous()

    def _normalize(self, rows: Tensor, weight: Tensor, bias: Tensor, out: Tensor) -> None:
        out.copy_(F.layer_norm(rows, (self.config.d_model,), weight, bias, self.config.norm_eps))

    def _layer_views(self, l: int) -> SimpleNamespace:
        """What a step hands the operators of layer ``l``: indexing the stacked tensors once a step costs more
        host time than launching on them."""
        w, q, last = self.w, self.query if self.fused else self.query[l], l + 1 == self.config.layers
        following = (w["final_norm_w"], w["final_norm_b"]) if last else (w["input_norm_w"][l + 1], w["input_norm_b"][l + 1])
        return SimpleNamespace(
            query=q, w_query=w["w_query"][l], next_query=None if last else w["w_query"][l + 1],
            selection=(q[:, 0:64], self.anchor_keys[l], q[:, 64:128], self.router_stats[0][l], self.router_stats[1][l],
                       w["anchor_gamma"][l], w["anchor_bias"][l], q[:, 128:256], self.partner_anchor_cache[l],
                       self.partner_keys[l], self.router_stats[2][l], self.router_stats[3][l], w["partner_gamma"][l],
                       w["partner_bias"][l]),
            caches=(self.expanded_cache[l], self.operand_cache[l]),
            first_layer=(w["anchor_weight"][l], w["partner_weight"][l], w["product_weight"][l], w["first_bias"][l]),
            second_layer=(w["w2"][l], w["b2"][l]), relation_norm=(w["relation_norm_w"][l], w["relation_norm_b"][l]),
            w_query_t=w["w_query"][l].t(), mix=w["mix"][l], next_norm=following)

    def _step_fused(self, tokens: Tensor, boundaries: Tensor, keep_selection: bool, advance: bool = True,
                    greedy: bool = False, chosen_out: Tensor | None = None):
        """The same step with the elementwise glue folded into the library's kernels:
        1 launch per layer where the selector fits in front of the single-launch relation tail, 2
        (select, tail) where only the tail applies, otherwise up to 5
        (query projection, select, relation hidden, second MLP layer GEMM, norm-reduce + residual +
        next LayerNorm).  Every LayerNorm is
        computed by the kernel that produces its input (the embedding, the residual update) and
        handed on as a 16-bit matrix, so the projections are plain tensor-core GEMMs."""
        cfg, w = self.config, self.w
        pos = self.position
        tokens, boundaries = tokens.contiguous(), boundaries.contiguous()
        if self.prefetch:
            main = torch.cuda.current_stream(self.device)
            self._side_stream.wait_stream(main)
            with torch.cuda.stream(self._side_stream):
                # in the order the step reads them
                l2_prefetch([w["anchor_weight"], w["partner_weight"], self.anchor_keys, self.partner_keys,
                             *self.router_stats, self.partner_anchor_cache, w["product_weight"], w["w2"],
                             self.operand_cache, w["w_query"], self.head_weight])
        if self.fused_front:
            hidden, packed = decode_front(tokens, boundaries, w["token_embedding"], w["boundary_embedding"],
                                          w["position_embedding"], pos, self.input_scale, w["memory_norm_w"],
                                          w["memory_norm_b"], w["input_norm_w"][0], w["input_norm_b"][0], cfg.norm_eps,
                                          self.front_weight, w["w_packed"].shape[0], self.memory_normalized,
                                          self.normalized, self.query)
        else:
            hidden = decode_embed_norm(tokens, boundaries, w["token_embedding"], w["boundary_embedding"],
                                       w["position_embedding"], pos, self.input_scale,
                                       w["memory_norm_w"], w["memory_norm_b"], self.memory_normalized,
                                       w["input_norm_w"][0], w["input_norm_b"][0], self.normalized, cfg.norm_eps)
        if self.fused_front:
            sparse_cache_append(packed, self.anchor_keys, self.partner_keys, self.operand_cache,
                                self.partner_anchor_cache, *self.router_caches, *self.router_stats,
                                w["anchor_conv_weight"], w["partner_conv_weight"], pos, cfg.block_size)
        elif self.append_in_projection:
            # the packed projection's epilogue writes the token caches and updates the router state
            packed = packed_projection_append(self.memory_normalized, w["w_packed"], self.anchor_keys,
                                              self.partner_keys, self.operand_cache, self.partner_anchor_cache,
                                              *self.router_caches, *self.router_stats, w["anchor_conv_weight"],
                                              w["partner_conv_weight"], pos, cfg.block_size)
        else:
            packed = self._project(self.memory_normalized, w["w_packed"])
            sparse_cache_append(packed, self.anchor_keys, self.partner_keys, self.operand_cache,
                                self.partner_anchor_cache, *self.router_caches, *self.router_stats,
                                w["anchor_conv_weight"], w["partner_conv_weight"], pos, cfg.block_size)
        if self.stacked_expand and not self.append_in_projection and (self.fused_front or cfg.d_model <= 512):
            # every layer's operand row of this position is known: expand them all at once, straight from
            # the packed rows (written two launches back), so that this launch overlaps the append (us a step,
            # from the operand cache -> from the packed rows: 24 sequences of d 256, 4 layers 89.0 -> 86.1, 32 of d 512,
            # 6 layers 159.7 -> 158.0; of d 768, 12 layers, where the two compete for memory, 8 256.1 -> 257.3, 28 386.1 -> 388.9).
            # It reads `packed` ahead of its dependency wait: exactly one launch, which waits before it lets this one go, has
            # to lie between the projection and this call: the append.
            expanded_cache_append_packed(self.expanded_cache, packed, w["anchor_weight"], w["partner_weight"],
                                         w["first_bias"], pos)
        elif self.stacked_expand:
            expanded_cache_append(self.expanded_cache, self.operand_cache, w["anchor_weight"],
                                  w["partner_weight"], w["first_bias"], pos)
        if keep_selection:
            self.last_selection = []
        trace = self.trace
        if trace is not None:
            trace.append({"stage": "append", "embedded": hidden.clone(), "packed": packed.clone(),
                          "memory_normalized": self.memory_normalized.clone(),
                          "normalized": self.normalized.clone()})
        K = cfg.k_max
        for l in range(cfg.layers):
            # layer 0 projects the embedding's normalised rows; later layers find their queries
            # written by the previous layer's norm-reduce when that fusion is on
            layer, last = self._layers[l], l + 1 == cfg.layers
            next_w, next_b = layer.next_norm
            if (self.fused_query or self.layer_tail) and (l > 0 or self.fused_front):
                q, selection = self.query, layer.selection
            else:
                q = self._project(self.normalized, layer.w_query)
                selection = (q[:, 0:64], *layer.selection[1:2], q[:, 64:128], *layer.selection[3:7], q[:, 128:256],
                             *layer.selection[8:])
            if self.whole_layer:
                if trace is not None:
                    entry = {"stage": "layer", "layer": l, "query": q.clone(), "hidden_before": hidden.clone()}
                    trace.append(entry)
                anchor, _, partner, partner_score = relation_layer(
                    *selection, pos, cfg.local_window, cfg.top_blocks, K, cfg.strict_valid,
                    *layer.caches, layer.first_layer[2], *layer.second_layer, *layer.relation_norm, cfg.norm_eps, hidden,
                    layer.mix, next_w, next_b, cfg.norm_eps, self.normalized, layer.next_query,
                    None if last else self.query)
                if trace is not None:
                    entry.update(anchor=anchor.clone(), partner=partner.clone(), partner_score=partner_score.clone(),
                                 hidden_after=hidden.clone(), next_normalized=self.normalized.clone())
                    if not last:
                        entry["next_query"] = self.query.clone()
                if keep_selection:
                    self.last_selection.append((anchor, partner))
                continue
            anchor, _, partner, partner_score = relation_select_packed(
                *selection, pos, cfg.local_window, cfg.top_blocks, K, cfg.strict_valid)
            if trace is not None:
                entry = {"stage": "layer", "layer": l, "query": q.clone(), "anchor": anchor.clone(),
                         "partner": partner.clone(), "partner_score": partner_score.clone(),
                         "hidden_before": hidden.clone()}
                trace.append(entry)
            if self.layer_tail:
                self._tail(*layer.caches, anchor, partner, partner_score, layer.first_layer[2],
                           *layer.second_layer, *layer.relation_norm, pos, cfg.norm_eps, hidden, layer.mix,
                           next_w, next_b, cfg.norm_eps, self.normalized, layer.next_query,
                           None if last else self.query)
                if trace is not None:
                    entry.update(hidden_after=hidden.clone(), next_normalized=self.normalized.clone())
                    if not last:
                        entry["next_query"] = self.query.clone()
                if keep_selection:
                    self.last_selection.append((anchor, partner))
                continue
            if self.stacked_expand:
                relation_hidden_cached_out(self.relation_hidden, *layer.caches, anchor, partner, layer.first_layer[2])
            else:
                relation_hidden_cache_update_out(self.relation_hidden, *layer.caches, anchor, partner, *layer.first_layer,
                                                 pos)
            if self.fused_tail:
                relation_tail(self.relation_hidden, w["w2"][l], w["b2"][l], partner_score,
                              w["relation_norm_w"][l], w["relation_norm_b"][l], pos, cfg.norm_eps,
                              hidden, w["mix"][l])
                layer_norm_cast(hidden, next_w, next_b, cfg.norm_eps, self.normalized)
            elif self.second_layer_splits > 1:
                # few rows, long reduction: split-K tensor-core GEMM, its fp32 slices summed by norm-reduce
                slices = packed_projection_slices(self.relation_hidden.view(-1, self.relation_hidden.size(-1)),
                                                  w["w2"][l], self.second_layer_splits)
                relation_norm_reduce_residual_norm_slices(
                    slices.view(self.second_layer_splits, -1, K, cfg.d_model), self.b2_f32[l], partner_score,
                    w["relation_norm_w"][l], w["relation_norm_b"][l], pos, cfg.norm_eps, hidden, w["mix"][l],
                    next_w, next_b, cfg.norm_eps, self.normalized)
            else:
                raw = F.linear(self.relation_hidden, *layer.second_layer)               # [B, K, d]
                if trace is not None:
                    entry["raw"] = raw.clone()
                if self.fused_query and not last:
                    relation_norm_reduce_residual_norm_project(
                        raw, partner_score, *layer.relation_norm, pos, cfg.norm_eps, hidden, layer.mix, next_w, next_b,
                        cfg.norm_eps, self.normalized, layer.next_query, self.query)
                else:
                    relation_norm_reduce_residual_norm(raw, partner_score, *layer.relation_norm, pos, cfg.norm_eps, hidden,
                                                       layer.mix, next_w, next_b, cfg.norm_eps, self.normalized)
            if trace is not None:
                entry.update(relation_hidden=self.relation_hidden.clone(), hidden_after=hidden.clone(),
                             next_normalized=self.normalized.clone())
                if self.fused_query and not last:
                    entry["next_query"] = self.query.clone()
            if keep_selection:
                self.last_selection.append((anchor, partner))
        self.last_final = self.normalized
        if greedy:
            # head projection + greedy arg-max + position increment in one launch
            if chosen_out is not None:
                chosen = chosen_out
                logits = skinny_projection_greedy_into(self.normalized, self.head_weight, self.head_bias,
                                                       cfg.vocab_size, self.argmax_scratch, pos, chosen_out)
            else:
                logits, chosen = skinny_projection_greedy(self.normalized, self.head_weight, self.head_bias,
                                                          cfg.vocab_size, self.argmax_scratch, pos)
            self.last_logits = logits
            if self.prefetch:
                main.wait_stream(self._side_stream)      # join the side branch (long finished) at the step's end
            return chosen
        logits = self._project(self.normalized, self.head_weight, self.head_bias)
        if self.prefetch:
            main.wait_stream(self._side_stream)
        self.last_logits = logits                        # [B, padded vocab + boundary vocab]
        token_logits = logits[:, :cfg.vocab_size]
        boundary_logits = logits[:, cfg.vocab_size:cfg.vocab_size + cfg.boundary_vocab_size]
        if advance:
            pos.add_(1)
        return token_logits, boundary_logits

    # ------------------------------------------------------------------ CUDA graph
    def capture(self) -> None:
        """Capture one ``step`` into a CUDA graph with static input / output buffers.  State and
        position are left exactly as they were."""
        B = self.batch
        self.static_tokens = torch.zeros(B, device=self.device, dtype=torch.int64)
        self.static_boundaries = torch.zeros(B, device=self.device, dtype=torch.int64)
        saved = int(self.position.item())
        stream = torch.cuda.Stream(self.device)
        stream.wait_stream(torch.cuda.current_stream(self.device))
        with torch.cuda.stream(stream):
            for _ in range(2):                                   # warm-up outside capture
                self.step_greedy(self.static_tokens, self.static_boundaries)
                self.position.fill_(saved)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                if self.fused:
                    self.static_next = self.step_greedy(self.static_tokens, self.static_boundaries)
                    V, Vb = self.config.vocab_size, self.config.boundary_vocab_size
                    self.static_token_logits = self.last_logits[:, :V]
                    self.static_boundary_logits = self.last_logits[:, V:V + Vb]
                else:
                    self.static_token_logits, self.static_boundary_logits = self.step(
                        self.static_tokens, self.static_boundaries)
                    self.static_next = self.static_token_logits.argmax(-1)
        torch.cuda.current_stream(self.device).wait_stream(stream)
        self.position.fill_(saved)
        self._graph = graph

    def replay(self) -> None:
        self._graph.replay()

    def capture_host_io(self, mapped: bool | None = None) -> None:
        """Capture the greedy step together with its host transfers, so that a serving loop pays one
        graph launch and one stream synchronisation per position (``step_host``): it writes the token
        and boundary ids into the pinned tensors ``host_tokens`` / ``host_boundaries`` ``[B]`` (int64; the
        two rows of ``host_ids``, copied to the device by one node at the head of the graph) and finds the
        chosen tokens in the pinned ``host_next``.  ``mapped`` (default: whenever the head projection's
        greedy launch applies): the head kernel writes the choices into the pinned memory itself, through
        a device view of ``host_next``, instead of a copy node at the tail of the graph.  (Reading the ids
        through such a view was measured too: it puts a host-memory round trip at the start of the step's
        dependency chain and is 10-20 us slower than the copy.)  State and position are left exactly as
        they were."""
        B = self.batch
        self.host_ids = torch.zeros(2, B, dtype=torch.int64).pin_memory()
        self.host_tokens, self.host_boundaries = self.host_ids[0], self.host_ids[1]
        self.host_next = torch.zeros(B, dtype=torch.int64).pin_memory()
        can_map = self.fused and self.skinny
        mapped = can_map if mapped is None else (bool(mapped) and can_map)
        ids = torch.zeros(2, B, device=self.device, dtype=torch.int64)
        tokens, boundaries = ids[0], ids[1]
        chosen_view = None
        if mapped:
            try:
                chosen_view = mapped_host_view(self.host_next, self.device)
            except (RuntimeError, TypeError, ValueError):      # no device view of pinned memory here: copy node
                mapped = False
        saved = int(self.position.item())
        stream = torch.cuda.Stream(self.device)
        stream.wait_stream(torch.cuda.current_stream(self.device))
        with torch.cuda.stream(stream):
            for _ in range(2):                                   # warm-up outside capture
                self.step_greedy(tokens, boundaries, chosen_view)
                self.position.fill_(saved)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                ids.copy_(self.host_ids, non_blocking=True)
                chosen = self.step_greedy(tokens, boundaries, chosen_view)
                if not mapped:
                    self.host_next.copy_(chosen, non_blocking=True)
        torch.cuda.current_stream(self.device).wait_stream(stream)
        self.position.fill_(saved)
        self.host_io_mapped = mapped
        self._host_graph, self._host_graph_buffers = graph, (ids, chosen)

    def step_host(self) -> Tensor:
        """One position through the graph of ``capture_host_io``: reads ``host_tokens`` /
        ``host_boundaries``, returns ``host_next`` (valid on return: the stream is synchronised)."""
        self._host_graph.replay()
        torch.cuda.current_stream(self.device).synchronize()
        return self.host_next
