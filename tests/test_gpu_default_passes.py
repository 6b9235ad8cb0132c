"""The whole-sequence passes as a program calls them, without `keep`: the fused relation MLP's path."""
from __future__ import annotations

import torch

import pytest

from gpu_util import assert_status_clear

pytestmark = pytest.mark.gpu


def _layer(dtype=torch.bfloat16, seed=3, **sizes):
    from relation_lm.inference.prefill import RoutedPrefillLayer
    from relation_lm.inference.routed_model import RoutedRelationConfig, RoutedRelationLM

    cfg = RoutedRelationConfig(**{**dict(vocab_size=32, boundary_vocab_size=4, d_model=256, layers=1, max_context=128, block_size=16,
                                         local_window=32, top_blocks=2), **sizes})
    return RoutedPrefillLayer(RoutedRelationLM(cfg, seed=seed), 0, "cuda", dtype)


def _rows(batch, length, d, seed=5):
    return torch.randn(batch, length, d, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def test_prefill_takes_rows_of_a_wider_tensor():
    """Residual rows with a row stride of their own, as a column slice has them."""
    layer = _layer()
    x = _rows(2, 128, 320)[..., :256]
    assert not x.is_contiguous()
    state = layer.build_state(x)
    dense = layer.build_state(x.contiguous())
    assert all(torch.equal(state[n], dense[n]) for n in state)
    assert torch.equal(layer.forward(x, state), layer.forward(x.contiguous(), state))
    assert_status_clear()


@pytest.mark.parametrize("block", [448, 512])
def test_prefill_of_blocks_beyond_the_state_kernels_tile(block):
    layer = _layer(max_context=2 * block, block_size=block, local_window=48, top_blocks=1)
    x = _rows(2, 2 * block, 256)
    state, keep = layer.build_state(x), {}
    kept = layer.forward(x, state, keep)
    # one selection on both sides, the relation MLP in one kernel or three: its rounding steps (see test_gpu_relation_mlp)
    assert float((layer.forward(x, state) - kept).abs().max()) <= 2 * 2 ** -8 * float(keep["context"].abs().max().clamp_min(1.0))
    assert_status_clear()


def test_only_the_first_launch_of_a_composition_is_ordinary():
    from relation_lm.kernels import _abi
    from relation_lm.kernels.packed_projection import layer_norm_cast

    x, w = _rows(1, 4, 64).view(4, 64), torch.ones(64, device="cuda")
    assert _abi.LIB.rlm_set_programmatic_launch(2) == 0
    layer_norm_cast(x, w, w, 1e-5, torch.empty_like(x))
    assert _abi.LIB.rlm_set_programmatic_launch(0) == 1
    assert_status_clear()


def _step(dtype):
    """The bound of test_gpu_relation_mlp: one rounding step of the largest term, within twice the largest value."""
    return 2 * (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)


@pytest.mark.parametrize("dtype,sizes", [
    (torch.bfloat16, {}), (torch.float16, {"max_context": 192, "k_max": 4}), (torch.bfloat16, {"d_model": 768, "strict_valid": True}),
    (torch.float16, {"d_model": 512, "top_blocks": 4, "block_size": 32}), (torch.bfloat16, {"k_max": 6}),          # K 6: three kernels
])
def test_prefill_equals_its_form_of_separate_kernels(dtype, sizes):
    _prefill_equals_separate_kernels(dtype, sizes, 3)


def test_prefill_of_eight_long_contexts_equals_its_form_of_separate_kernels():
    _prefill_equals_separate_kernels(torch.bfloat16, dict(d_model=512, max_context=4096, block_size=64, local_window=128, top_blocks=4), 8)


def _prefill_equals_separate_kernels(dtype, sizes, batch):
    """From the same state and rows: one selection on both sides, values within the relation MLP's rounding steps."""
    layer = _layer(dtype, **sizes)
    cfg = layer.config
    assert layer.fused_mlp == (cfg.k_max != 6)
    x = _rows(batch, cfg.max_context, cfg.d_model)
    state, keep = layer.build_state(x), {}
    kept, out = layer.forward(x, state, keep), layer.forward(x, state)
    assert float((out - kept).abs().max()) <= _step(dtype) * float(keep["context"].abs().max().clamp_min(1.0)) * float(layer.w["mix"])
    assert torch.equal(out, layer.forward(x, state))                                    # and it repeats itself
    assert_status_clear()


def _stack(dtype, **sizes):
    from relation_lm.inference.multi_anchor import MultiAnchorConfig, MultiAnchorPrefill, MultiAnchorRoutedStack

    cfg = MultiAnchorConfig(**{**dict(d_model=256, anchors_per_block=4, partners_per_anchor=4, depth=2, max_context=192, block_size=16,
                                      local_window=32, top_blocks=2), **sizes})
    return MultiAnchorPrefill(MultiAnchorRoutedStack(cfg, seed=7), "cuda", dtype)


@pytest.mark.parametrize("dtype,slots,d", [(torch.bfloat16, 4, 256), (torch.float16, 2, 256), (torch.bfloat16, 3, 256),
                                           (torch.bfloat16, 4, 512), (torch.float16, 3, 512)])
def test_multi_anchor_equals_its_form_of_separate_kernels(dtype, slots, d):
    _multi_anchor_equals_separate_kernels(dtype, slots, d, 2, 192)


def test_multi_anchor_of_long_contexts_equals_its_form_of_separate_kernels():
    _multi_anchor_equals_separate_kernels(torch.bfloat16, 4, 512, 16, 2048, block_size=32, local_window=64, top_blocks=3)


def _multi_anchor_equals_separate_kernels(dtype, slots, d, batch, length, **sizes):
    """Layer by layer from the same residual stream (over several layers a rounding may decide a near tie), then the
    whole pass as the chain of its layers: entry of the first one from its source, and the final LayerNorm."""
    stack = _stack(dtype, anchors_per_block=slots, d_model=d, max_context=length, **sizes)
    assert stack.fused_mlp and stack.fused_mix == (slots != 3)                          # three slots: mixed on their own
    hidden, memory = _rows(batch, length, d), _rows(batch, length, d, seed=6).to(dtype)
    stream = hidden.clone()
    for layer in range(2):
        state, keep = stack.build_state(layer, memory), {}
        kept = stack.forward_layer(layer, stream.clone(), state, keep)
        out = stack.forward_layer(layer, torch.empty_like(stream), state, source=stream)
        assert torch.equal(out, stack.forward_layer(layer, stream.clone(), state))
        bound = _step(dtype) * float(keep["slot_context"].abs().max().clamp_min(1.0)) * float(stack.layers[layer]["gate"])
        assert float((out - kept).abs().max()) <= bound
        stream = out
    want = torch.nn.functional.layer_norm(stream, (d,), stack.final_norm_w, stack.final_norm_b, stack.config.norm_eps)
    got = stack.forward(hidden, memory)
    # fp32 sums of d terms in another order
    assert float((got - want).abs().max()) <= 1.0e-5 * float(want.abs().max())
    assert_status_clear()


def test_programmatic_launch_leaves_a_pass_as_it_is():
    """The same pass with every launch in the ordinary way: `build_state` and `forward` without their decorator."""
    layer, stack = _layer(), _stack(torch.bfloat16)
    x, memory = _rows(2, 128, 256), _rows(2, 192, 256, seed=6).bfloat16()
    plain = type(layer).forward.__wrapped__(layer, x, type(layer).build_state.__wrapped__(layer, x))
    hidden = _rows(2, 192, 256)
    state = type(stack).build_state.__wrapped__(stack, 0, memory)
    slots = type(stack).forward_layer.__wrapped__(stack, 0, hidden.clone(), state)
    for _ in range(20):
        assert torch.equal(layer.forward(x, layer.build_state(x)), plain)
        assert torch.equal(stack.forward_layer(0, hidden.clone(), stack.build_state(0, memory)), slots)
    assert_status_clear()


def test_a_captured_pass_replays_on_new_rows():
    layer = _layer(torch.float16)
    x = _rows(2, 128, 256)
    layer.forward(x, layer.build_state(x))                   # warm
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = layer.forward(x, layer.build_state(x))
    for seed in (8, 9):
        x.copy_(_rows(2, 128, 256, seed=seed))
        graph.replay()
        assert torch.equal(out, layer.forward(x, layer.build_state(x)))
    assert_status_clear()
