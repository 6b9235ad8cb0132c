"""A whole-sequence layer whose operators are called in two groups from native code, against the same operators called
one by one: the same bits, also where a call declines or the tiled selector does not fit."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear

pytestmark = pytest.mark.gpu


def _layer(dtype, **config):
    from relation_lm.inference.prefill import RoutedPrefillLayer
    from relation_lm.inference.routed_model import RoutedRelationConfig, RoutedRelationLM

    cfg = RoutedRelationConfig(vocab_size=64, boundary_vocab_size=8, layers=1, **config)
    return RoutedPrefillLayer(RoutedRelationLM(cfg, seed=3), 0, "cuda", dtype)


def _one_by_one(monkeypatch, layer, x):
    from relation_lm.kernels import _abi

    with monkeypatch.context() as m:
        m.setattr(_abi, "direct_call", lambda *a: NotImplemented)
        state = layer.build_state(x)
        return state, layer.forward(x, state)


def _watched(monkeypatch):
    """Which groups were called and whether they ran."""
    from relation_lm.kernels import _abi

    calls, direct_call = [], _abi.direct_call

    def watched(name, *args):
        made = direct_call(name, *args)
        calls.append((name, made is not NotImplemented))
        return made

    monkeypatch.setattr(_abi, "direct_call", watched)
    return calls


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,config", [
    (1, dict(d_model=256, max_context=512, block_size=16, local_window=32, top_blocks=2)),
    (3, dict(d_model=128, max_context=136, block_size=17, local_window=20, top_blocks=3, k_max=4, strict_valid=True)),
    (2, dict(d_model=768, max_context=128, block_size=64, local_window=128, top_blocks=1)),
])
def test_groups_equal_the_operators_one_by_one(monkeypatch, dtype, batch, config):
    layer = _layer(dtype, **config)
    x = torch.randn(batch, config["max_context"], config["d_model"], device="cuda")
    want_state, want = _one_by_one(monkeypatch, layer, x)
    calls = _watched(monkeypatch)
    state = layer.build_state(x)
    got = layer.forward(x, state)
    assert calls == [("prefill_state", True), ("prefill_layer", True)]
    assert list(state) == list(want_state) and all(torch.equal(state[k], want_state[k]) for k in state)
    assert got.shape == x.shape and torch.equal(got, want)
    # rows with a stride of their own: the same layer, one residual copy
    wide = torch.zeros(batch, config["max_context"], config["d_model"] + 4, device="cuda")
    wide[:, :, :config["d_model"]] = x
    assert torch.equal(layer.forward(wide[:, :, :config["d_model"]], state), want)
    # a derivative is asked for: the operators one by one, none of which has one
    del calls[:]
    asked = x.clone().requires_grad_()
    out = layer.forward(asked, layer.build_state(asked))
    assert calls == [("prefill_state", False), ("prefill_layer", False)] and torch.equal(out, want)
    with pytest.raises(RuntimeError, match="does not require grad"):
        out.sum().backward()
    assert_status_clear()


def test_a_selector_that_does_not_fit_falls_back(monkeypatch):
    from relation_lm.kernels import _abi

    config = dict(d_model=128, max_context=8192, block_size=16, local_window=32, top_blocks=2)     # 512 blocks
    layer, other = _layer(torch.bfloat16, **config), _layer(torch.bfloat16, **config)
    other.tiled_select = False
    x = torch.randn(1, 8192, 128, device="cuda")
    state = layer.build_state(x)
    calls = _watched(monkeypatch)
    before = _abi.launch_count()
    want = other.forward(x, state)
    launches = _abi.launch_count() - before
    assert torch.equal(layer.forward(x, state), want) and not layer.tiled_select
    assert calls == [("prefill_layer", True)] and _abi.launch_count() - before == 2 * launches       # nothing is run twice
    # an error of another operator of the group is the caller's, whatever it says, and turns nothing off
    small = _layer(torch.bfloat16, d_model=128, max_context=128, block_size=16, local_window=32, top_blocks=2)
    y = torch.randn(1, 128, 128, device="cuda")
    state_y = small.build_state(y)
    broken = dict(state_y, expanded_cache=state_y["expanded_cache"][:, :, 1:])
    with pytest.raises(ValueError):
        small.forward(y, broken)
    assert small.tiled_select
    with pytest.raises(ValueError):
        layer.forward(x.double(), state)
    assert_status_clear()
