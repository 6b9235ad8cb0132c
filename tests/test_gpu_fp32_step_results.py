"""What a single-precision step takes and returns, beside its values."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear

pytestmark = pytest.mark.gpu


def _decoder(batch):
    from relation_lm.inference.routed_model import RoutedRelationConfig, RoutedRelationLM
    from relation_lm.inference.stateful_decode import StatefulDecoder

    cfg = RoutedRelationConfig(vocab_size=50, boundary_vocab_size=6, d_model=64, layers=2, max_context=32, block_size=8,
                               local_window=8, top_blocks=1)
    return StatefulDecoder(RoutedRelationLM(cfg, seed=1), batch, "cuda", torch.float32)


@pytest.mark.parametrize("batch", [1, 3])
def test_results_belong_to_their_step(batch):
    dec = _decoder(batch)
    tokens, bounds = (torch.randint(0, n, (4, batch), device="cuda") for n in (50, 6))
    kept, copies = [], []
    for t in range(4):
        results = (*dec.step(tokens[t], bounds[t]), dec.last_final)
        assert results[0].is_contiguous() and results[1].is_contiguous()
        assert results[0].shape == (batch, 50) and results[1].shape == (batch, 6)
        kept.append(results)
        copies.append([r.clone() for r in results])
    assert all(torch.equal(a, b) for k, c in zip(kept, copies) for a, b in zip(k, c))
    assert not torch.equal(kept[0][2], kept[1][2])
    assert_status_clear()


@pytest.mark.parametrize("batch", [1, 3])
def test_ids_as_an_embedding_takes_them(batch):
    """32-bit ids, and one id for all sequences."""
    tokens = torch.arange(batch, device="cuda") + 7
    for other in (torch.tensor([2], device="cuda"), torch.tensor(2, device="cuda"),
                  torch.full((batch,), 2, device="cuda", dtype=torch.int32)):
        want, got = _decoder(batch), _decoder(batch)
        a = want.step(tokens, torch.full((batch,), 2, device="cuda"))
        b = got.step(tokens.int(), other)
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    dec = _decoder(batch)
    with pytest.raises(ValueError):
        dec.step(tokens.view(batch, 1), tokens.view(batch, 1))
    assert_status_clear()


@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("keep_selection", [False, True])
def test_a_step_past_the_context_is_reported_and_changes_no_state(batch, keep_selection):
    """Every kernel of that step still waits for its predecessor, so that the steps around it are what they are without
    programmatic launch."""
    from relation_lm.kernels import _abi

    results = []
    for early in (False, True):
        dec = _decoder(batch)
        dec.programmatic_launch = early
        tokens, bounds = (torch.randint(0, n, (40, batch), generator=torch.Generator().manual_seed(n)).cuda() for n in (50, 6))
        for t in range(32):
            dec.step(tokens[t], bounds[t], keep_selection)
        assert_status_clear()
        names = ("anchor_keys", "partner_keys", "operand_cache", "partner_anchor_cache", "expanded_cache")
        state = [getattr(dec, n).clone() for n in names] + [s.clone() for s in dec.router_caches + dec.router_stats]
        dec.step(tokens[32], bounds[32], keep_selection)
        assert _abi.read_status() != 0
        now = [getattr(dec, n) for n in names] + dec.router_caches + dec.router_stats
        assert all(torch.equal(a, b) for a, b in zip(state, now))
        dec.slide(1)
        dec.position.fill_(24)
        results.append([r.clone() for t in range(33, 40) for r in dec.step(tokens[t], bounds[t], keep_selection)])
        assert_status_clear()
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("batch", [1, 2])
def test_weights_that_start_anywhere(batch):
    """The heads' weights are the model's own where those are already on the device in single precision: slices of a flat
    buffer, off a 16-byte boundary, included."""
    from relation_lm.inference.routed_model import RoutedRelationConfig, RoutedRelationLM
    from relation_lm.inference.stateful_decode import StatefulDecoder

    cfg = RoutedRelationConfig(vocab_size=50, boundary_vocab_size=6, d_model=64, layers=1, max_context=32, block_size=8,
                               local_window=8, top_blocks=1)
    model = RoutedRelationLM(cfg, seed=1).cuda()
    want = StatefulDecoder(model, batch, "cuda", torch.float32)
    for weight in (model.token_embedding.weight, model.boundary_output.weight):
        flat = torch.cat((weight.detach().new_zeros(1), weight.detach().flatten()))
        weight.data = flat[1:].view_as(weight)
    got = StatefulDecoder(model, batch, "cuda", torch.float32)
    tokens, bounds = (torch.randint(0, n, (4, batch), device="cuda") for n in (50, 6))
    for t in range(4):
        a, b = want.step(tokens[t], bounds[t]), got.step(tokens[t], bounds[t])
        # a sum of 64 products in another order: 64 roundings of a sum of magnitudes below 64 times the largest product
        for x, y in zip(a, b):
            assert float((x - y).abs().max()) <= 64 * 2.0 ** -24 * 64 * float(want.last_final.abs().max())
    assert torch.equal(want.position, got.position) and torch.equal(want.expanded_cache, got.expanded_cache)
    assert_status_clear()


@pytest.mark.parametrize("batch,vocab", [(1, 24_100), (5, 40_100), (4, 40_100)])
def test_heads_of_many_columns(batch, vocab):
    """On either side of where a library's product takes the heads: both heads against 64-bit products of the step's rows."""
    from relation_lm.inference.routed_model import RoutedRelationConfig, RoutedRelationLM
    from relation_lm.inference.stateful_decode import StatefulDecoder

    cfg = RoutedRelationConfig(vocab_size=vocab, boundary_vocab_size=6, d_model=264, layers=1, max_context=32, block_size=8,
                               local_window=8, top_blocks=1)
    dec = StatefulDecoder(RoutedRelationLM(cfg, seed=1), batch, "cuda", torch.float32)
    assert dec.few_rows and dec.few_heads == (batch == 4)
    for keep_selection in (False, True):
        heads = dec.step(torch.arange(batch, device="cuda"), torch.zeros(batch, dtype=torch.int64, device="cuda"), keep_selection)
        rows = dec.last_final.double()
        for got, (weight, bias) in zip(heads, ((dec.w["token_embedding"], None), (dec.w["boundary_w"], dec.w["boundary_b"]))):
            full = torch.nn.functional.linear(rows, weight.double(), bias.double() if bias is not None else None)
            size = rows.abs() @ weight.double().abs().T + 1.0
            assert got.is_contiguous() and bool(((got.double() - full).abs() <= 264 * 2.0 ** -24 * size).all())
    assert int(dec.position) == 2
    assert_status_clear()
