"""Relation hidden states of a few sequences in single precision against an evaluation in 64 bits, at the edges of the
kernel's range (one partner to eight, relation widths below a warp's 128, ragged hidden widths, many sequences a CTA)."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _inputs(B, T, R, H, K, t, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s, scale=1.0: torch.randn(*s, generator=g, device="cuda") * scale  # noqa: E731
    x = {"expanded": rand(B, T, 2 * H), "operand": rand(B, T, R), "anchor_w": rand(H, R, scale=R ** -0.5),
         "partner_w": rand(H, R, scale=R ** -0.5), "product_w": rand(H, R, scale=R ** -0.5), "bias": rand(H),
         "anchor": torch.randint(0, t + 1, (B,), generator=g, device="cuda", dtype=torch.int32),
         "partner": torch.randint(-3, T + 3, (B, K), generator=g, device="cuda", dtype=torch.int32)}
    x["anchor"][::3] = t                  # the position's own row, as anchor and as partner
    x["partner"][:, 0] = t
    return x


def _reference(x, t, update):
    """(hidden states, bound of their error, expanded cache) in 64 bits."""
    d = {k: v.double() if v.is_floating_point() else v.long() for k, v in x.items()}
    B, K = d["partner"].shape
    T, H = d["operand"].shape[1], d["product_w"].shape[0]
    rows = torch.arange(B, device="cuda")
    expanded = d["expanded"].clone()
    if update:
        cur = d["operand"][:, t]
        expanded[:, t, :H] = cur @ d["anchor_w"].T + d["bias"]
        expanded[:, t, H:] = cur @ d["partner_w"].T
    a, p = d["anchor"].clamp(0, T - 1), d["partner"].clamp(0, T - 1)
    prod = d["operand"][rows, a][:, None] * d["operand"][rows[:, None], p]
    z = prod @ d["product_w"].T + expanded[rows, a, :H][:, None] + expanded[rows[:, None], p, H:]
    # at most 16 roundings on the way of a term: four chained, five levels, the products and the two added terms; an
    # own row's sum has as many of its own.  GELU's slope is below 1.13, erff is good to a few units in the last place.
    size = prod.abs() @ d["product_w"].abs().T + expanded[rows, a, :H].abs()[:, None] + expanded[rows[:, None], p, H:].abs()
    if update:
        own = d["operand"][:, t].abs() @ (d["anchor_w"].abs() + d["partner_w"].abs()).T + d["bias"].abs()
        size = size + own[:, None]
    return torch.nn.functional.gelu(z), 1.13 * 16 * EPS * size + 8 * EPS * z.abs(), expanded


@pytest.mark.parametrize("update", [True, False])
@pytest.mark.parametrize("B,T,R,H,K", [
    (1, 128, 128, 1024, 8), (1, 40, 16, 37, 1), (3, 64, 48, 130, 5), (7, 96, 128, 2304, 8), (2, 32, 64, 64, 4),
    (12, 64, 128, 2304, 8), (33, 64, 128, 256, 8), (48, 32, 128, 3072, 3), (49, 32, 128, 64, 8), (2, 32, 144, 96, 8),
    (2, 32, 128, 96, 9),
    # both sides of the lines of sequences x hidden width (with the update | without) for narrower relations
    (12, 32, 96, 1024, 4), (13, 32, 96, 1024, 4), (32, 32, 96, 1024, 2), (33, 32, 96, 1024, 2), (24, 32, 64, 1024, 8), (25, 32, 64, 1024, 8),
    (9, 32, 32, 1024, 8), (10, 32, 32, 1024, 8), (12, 32, 16, 1024, 1), (13, 32, 16, 1024, 1), (12, 32, 128, 2048, 8), (12, 32, 128, 2052, 8),
])
def test_against_64_bits(B, T, R, H, K, update):
    from relation_lm.kernels.relation_reduce import relation_hidden_cache_update, relation_hidden_cached

    t = T - 5
    x = _inputs(B, T, R, H, K, t, 100 * B + K)
    want, bound, expanded = _reference(x, t, update)
    if update:
        got = relation_hidden_cache_update(x["expanded"], x["operand"], x["anchor"], x["partner"], x["anchor_w"],
                                           x["partner_w"], x["product_w"], x["bias"], torch.tensor(t, device="cuda"))
        rel = (x["expanded"].double() - expanded).abs().max() / expanded.abs().max()
        assert rel < 16 * EPS * R ** 0.5
    else:
        got = relation_hidden_cached(x["expanded"], x["operand"], x["anchor"], x["partner"], x["product_w"])
    assert got.shape == (B, K, H)
    assert torch.all((got.double() - want).abs() <= bound)
    assert_status_clear()


def test_rows_that_are_not_finite_stay_with_their_partner():
    from relation_lm.kernels.relation_reduce import relation_hidden_cached

    x = _inputs(2, 32, 128, 96, 8, 20, 7)
    x["partner"] = torch.arange(16, device="cuda", dtype=torch.int32).view(2, 8)
    x["anchor"].fill_(30)
    want = relation_hidden_cached(x["expanded"], x["operand"], x["anchor"], x["partner"], x["product_w"])
    x["operand"][0, 3, 5], x["operand"][1, 9, 127] = float("inf"), float("nan")
    got = relation_hidden_cached(x["expanded"], x["operand"], x["anchor"], x["partner"], x["product_w"])
    keep = torch.ones(2, 8, dtype=torch.bool, device="cuda")
    keep[0, 3] = keep[1, 1] = False
    assert torch.equal(got[keep], want[keep]) and got[1, 1].isnan().all()
    assert_status_clear()
