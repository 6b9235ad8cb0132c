"""``few_rows_projection``: single-precision products of at most 64 rows, against 64-bit products of the same operands.

A sum of K products in fp32, K / 32 of them at most in one lane's chain and a tree over the lanes and warps behind it,
is off by at most (K / 32 + 10) roundings of the sum of the magnitudes."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear

pytestmark = pytest.mark.gpu


def _check(out, x, w, b):
    x, w = x.double(), w.double()
    bound = (x.size(1) / 32 + 10) * 2.0 ** -24 * (x.abs() @ w.abs().T + (b.double().abs() if b is not None else 0.0))
    want = x @ w.T + (b.double() if b is not None else 0.0)
    assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("rows", [1, 2, 3, 5, 8, 9, 16, 17, 64])
@pytest.mark.parametrize("d_in,n_out", [(4, 1), (124, 7), (128, 2), (260, 33), (576, 512), (1028, 300), (3072, 768), (256, 5000)])
def test_matches_64_bit_products(rows, d_in, n_out):
    from relation_lm.kernels.packed_projection import few_rows_projection, few_rows_projection_pair

    g = torch.Generator().manual_seed(1000 * rows + d_in)
    wide = torch.randn(rows, d_in + 8, generator=g).cuda()
    x = wide[:, 4:4 + d_in]                                   # rows with a stride of their own
    w, b = torch.randn(n_out, d_in, generator=g).cuda(), torch.randn(n_out, generator=g).cuda()
    room = torch.full((rows * n_out + 64,), 7.0, device="cuda")
    out = room[:rows * n_out].view(rows, n_out)
    few_rows_projection(out, x, w, b)
    _check(out, x, w, b)
    assert bool((room[rows * n_out:] == 7.0).all())
    out2, other = torch.empty(rows, 5, device="cuda"), torch.randn(5, d_in, generator=g).cuda()
    few_rows_projection_pair(out, out2, x, w, other, b[:1].expand(5).contiguous())
    _check(out, x, w, None)
    _check(out2, x, other, b[:1].expand(5))
    again = torch.empty_like(out)
    few_rows_projection(again, x, w)
    assert torch.equal(again, out)                            # and the order of the sums is fixed
    assert_status_clear()


def test_refuses_what_it_does_not_take():
    from relation_lm.kernels.packed_projection import few_rows_projection

    x, w = torch.randn(4, 16, device="cuda"), torch.randn(8, 16, device="cuda")
    out = torch.empty(4, 8, device="cuda")
    for bad in ((out.half(), x.half(), w.half()), (out, x[:, :12], w), (out[:2], x, w), (out, x[:, 1:13], w[:, :12].contiguous()),
                (torch.empty(65, 8, device="cuda"), torch.randn(65, 16, device="cuda"), w)):
        with pytest.raises(ValueError):
            few_rows_projection(*bad)


@pytest.mark.parametrize("batch,layers,strided", [(1, 1, False), (3, 3, True), (8, 2, False)])
def test_grouped_calls_are_the_single_ones(batch, layers, strided):
    """The single-precision step with its operators called in groups and one by one (as it does to keep the selections):
    logits, state, position and version counters alike."""
    from relation_lm.inference.routed_model import RoutedRelationConfig, RoutedRelationLM
    from relation_lm.inference.stateful_decode import StatefulDecoder

    cfg = RoutedRelationConfig(vocab_size=301, boundary_vocab_size=9, d_model=256, layers=layers, max_context=64, block_size=8,
                               local_window=16, top_blocks=2)
    model = RoutedRelationLM(cfg, seed=5)
    one, two = StatefulDecoder(model, batch, "cuda", torch.float32), StatefulDecoder(model, batch, "cuda", torch.float32)
    ids = torch.arange(40, device="cuda").view(20, 2)[:, 0] % 9
    for t in range(20):
        tokens, bounds = (ids[t] + torch.arange(batch, device="cuda") * 7) % 301, ids[t].expand(batch)
        if strided:
            tokens = torch.stack((tokens, tokens), 1)[:, 0]
        before = [x.position._version for x in (one, two)]
        a, b = one.step(tokens, bounds), two.step(tokens, bounds, keep_selection=True)
        assert all(torch.equal(x, y) and x.is_contiguous() for x, y in zip(a, b))
        assert [x.position._version for x in (one, two)] == [v + 1 for v in before]
    for name in ("anchor_keys", "partner_keys", "operand_cache", "partner_anchor_cache", "expanded_cache", "position", "last_final"):
        assert torch.equal(getattr(one, name), getattr(two, name)), name
        if name != "last_final":
            assert getattr(one, name)._version == getattr(two, name)._version, name
    for x, y in zip(one.router_caches + one.router_stats, two.router_caches + two.router_stats):
        assert torch.equal(x, y)
    assert_status_clear()
