"""Host-side behaviour of the whole-sequence passes."""
from __future__ import annotations

import torch

from relation_lm.inference.multi_anchor import MultiAnchorConfig, MultiAnchorPrefill, MultiAnchorRoutedStack
from relation_lm.inference.prefill import RoutedPrefillLayer
from relation_lm.inference.routed_model import RoutedRelationConfig, RoutedRelationLM
from relation_lm.kernels import _abi


def _layer(**sizes):
    cfg = RoutedRelationConfig(**{**dict(vocab_size=32, boundary_vocab_size=4, d_model=64, layers=1, max_context=32, block_size=8,
                                         local_window=8, top_blocks=1), **sizes})
    return RoutedPrefillLayer(RoutedRelationLM(cfg, seed=0), 0, "cpu")


def test_row_tables_belong_to_their_pass():
    """Every pass fills its own tables on its own stream (or in its own graph): none is handed from one to the next."""
    layer = _layer()
    first, second = layer.rows(2, 32), layer.rows(2, 32)
    for a, b in zip(first, second):
        assert torch.equal(a, b) and a.data_ptr() != b.data_ptr()


def test_a_stack_without_layers_is_its_final_norm():
    stack = MultiAnchorRoutedStack(MultiAnchorConfig(d_model=64, depth=0), seed=0)
    hidden = torch.randn(2, 5, 64, generator=torch.Generator().manual_seed(1))
    out = MultiAnchorPrefill(stack, "cpu").forward(hidden, hidden.bfloat16())
    assert torch.equal(out, torch.nn.functional.layer_norm(hidden, (64,), stack.final_norm.weight, stack.final_norm.bias, 1e-5))


def test_a_composition_starts_with_an_ordinary_launch():
    """The kernel before it is the caller's and may still be writing weights; a part of a composition, or one inside a
    region that has switched programmatic launch on, takes the setting it finds."""
    setting = _abi.LIB.rlm_set_programmatic_launch

    def read():
        value = setting(0)
        setting(value)
        return value

    seen = []
    inner = _abi.programmatic_launch(first=False)(lambda: seen.append(read()))

    @_abi.programmatic_launch(first=False)
    def outer():
        seen.append(read())
        inner()
        setting(1)                       # as the first launch leaves it
        inner()
        seen.append(read())

    assert read() == 0
    outer()
    assert seen == [2, 2, 1, 1] and read() == 0
    previous = setting(1)
    inner()
    assert seen[-1] == 1 and setting(previous) == 1
    _abi.programmatic_launch(lambda: seen.append(read()))()
    assert seen[-1] == 1 and read() == 0
