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
