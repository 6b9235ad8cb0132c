"""The one-launch relation MLP of a whole-sequence pass against a plain fp32 PyTorch evaluation of the
same formulas (operands rounded where the kernel rounds: the products, the hidden states and the second layer's rows)."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear

pytestmark = pytest.mark.gpu


def _case(dtype, batch, length, slots, k, rdim, d, seed, hidden=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s, scale=1.0: torch.randn(*s, generator=g, device="cuda") * scale  # noqa: E731
    H, N = hidden or 4 * d, batch * length
    x = {
        "expanded": rn(batch, length, 2 * H, scale=0.5).to(dtype), "operand": rn(batch, length, rdim).to(dtype),
        "anchor": torch.randint(-1, length, (N, slots), generator=g, device="cuda", dtype=torch.int32),
        "partner": torch.randint(-3, length, (N, slots, k), generator=g, device="cuda", dtype=torch.int32),
        "score": rn(N, slots, k, scale=2.0), "active": torch.rand(N, slots, generator=g, device="cuda") < 0.8,
        "slot_weight": torch.softmax(rn(slots), 0), "scale": rn(1).abs(), "wm": rn(H, rdim, scale=rdim ** -0.5).to(dtype),
        "w2": rn(d, H, scale=H ** -0.5).to(dtype), "b2": rn(d, scale=0.1), "nw": 1 + rn(d, scale=0.1), "nb": rn(d, scale=0.1),
        "residual": rn(N, d),
    }
    x["score"][torch.rand(N, slots, k, generator=g, device="cuda") < 0.15] = -torch.inf
    return x


def _expected(x, length, limited, mixed):
    dtype = x["operand"].dtype
    N, S, K = x["score"].shape
    d = x["w2"].size(0)
    n = torch.arange(N, device="cuda")
    seq, t = n // length, n % length
    a = x["anchor"].long().clamp(0, length - 1)
    p = x["partner"].long().clamp(0, length - 1)
    out = torch.empty(N, d, device="cuda")
    wm, w2 = x["wm"].float(), x["w2"].float()
    H = wm.size(0)
    for lo in range(0, N, 256):
        r = slice(lo, min(N, lo + 256))
        op, ex = x["operand"][seq[r]].float(), x["expanded"][seq[r]].float()          # [n, T, .]
        rows = torch.arange(op.size(0), device="cuda")
        oa, ea = op[rows[:, None], a[r]], ex[rows[:, None], a[r]][..., :H]            # [n, S, .]
        pp = p[r].reshape(op.size(0), -1)
        opp = op[rows[:, None], pp].view(-1, S, K, op.size(-1))
        epp = ex[rows[:, None], pp][..., H:].reshape(-1, S, K, H)
        prod = (oa[:, :, None] * opp).to(dtype).float()
        hid = torch.nn.functional.gelu(prod @ wm.T + ea[:, :, None] + epp).to(dtype).float()
        raw = torch.nn.functional.layer_norm((hid @ w2.T + x["b2"]).to(dtype).float(), (d,), x["nw"], x["nb"], 1e-5)
        s = x["score"][r]
        live = torch.isfinite(s)
        if limited:
            limit = torch.ceil(torch.log2(t[r].double() + 2)).clamp(1, K)
            live &= torch.arange(K, device="cuda")[None, None] < limit[:, None, None]
        e = torch.where(live, torch.exp(s - torch.where(live, s, -1e4).amax(-1, keepdim=True)), 0.0)
        u = e / e.sum(-1, keepdim=True).clamp_min(1e-9)
        if mixed:
            w = torch.where(x["active"][r], x["slot_weight"], 0.0)
            u = u * (w / w.sum(-1, keepdim=True).clamp_min(1e-9))[..., None]
        out[r] = x["residual"][r] + x["scale"] * (u[..., None] * raw).sum((1, 2))
    return out


# d on both sides of one output part per cluster, tiles of one / several rows, ragged last tiles, every group size
@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16))
@pytest.mark.parametrize("batch,length,slots,k,rdim,d,limited", [
    (1, 3, 1, 8, 128, 512, True), (2, 37, 1, 8, 128, 512, True), (3, 50, 4, 4, 128, 512, False), (1, 129, 1, 4, 64, 256, True),
    (2, 33, 2, 8, 128, 256, False), (1, 70, 1, 8, 128, 768, True), (1, 21, 4, 8, 128, 768, False), (1, 40, 1, 4, 128, 64, True),
    (1, 19, 1, 16, 64, 384, True), (2, 45, 8, 4, 128, 128, False), (5, 700, 1, 8, 128, 512, True), (4, 900, 1, 8, 128, 256, True),
    (3, 600, 4, 4, 128, 512, False), (3, 800, 1, 8, 128, 768, True),
])
def test_matches_the_composition(dtype, batch, length, slots, k, rdim, d, limited):
    _check(dtype, batch, length, slots, k, rdim, d, 4 * d, limited)


# the fewest hidden units a CTA can have (two and three; d 64 .. 256 and 512: the wide form, 384 and 768: the other), with
# five tiles or more for every cluster: the first layer then runs two tiles ahead of the weights' last use
@pytest.mark.parametrize("batch,slots,k,rdim,d,hidden", [
    (56, 4, 8, 64, 64, 256), (56, 4, 8, 64, 64, 384), (56, 2, 16, 128, 256, 256), (28, 4, 8, 128, 512, 512),
    (28, 4, 8, 64, 512, 768), (56, 4, 8, 64, 384, 256), (28, 4, 8, 128, 768, 512), (28, 4, 8, 64, 768, 768),
])
def test_few_hidden_units_and_many_tiles(batch, slots, k, rdim, d, hidden):
    _check(torch.bfloat16, batch, 53, slots, k, rdim, d, hidden, False)


# one output part or two for widths that fit in one: 33 pairs of tiles (the most that are spread) and 34, and a hidden
# width that two parts cannot divide
@pytest.mark.parametrize("length,d,hidden", [(1056, 256, 1024), (1057, 256, 1024), (1056, 128, 512), (40, 256, 256), (300, 384, 1536)])
def test_tiles_over_one_or_two_parts(length, d, hidden):
    _check(torch.bfloat16, 1, length, 1, 8, 128, d, hidden, True)


def _check(dtype, batch, length, slots, k, rdim, d, hidden, limited):
    from relation_lm.kernels.relation_reduce import relation_mlp_rows, relation_mlp_rows_supported

    assert relation_mlp_rows_supported(k, slots, rdim, hidden, d, dtype)
    x = _case(dtype, batch, length, slots, k, rdim, d, d + 7 * k + length, hidden)
    mixed = slots > 1
    out = x["residual"].clone()
    relation_mlp_rows(out, x["expanded"], x["operand"], x["anchor"], x["partner"], x["score"], x["active"] if mixed else None,
                      x["slot_weight"] if mixed else None, x["scale"], x["wm"], x["w2"], x["b2"], x["nw"], x["nb"], 1e-5,
                      out, slots, length, limited)
    assert_status_clear()
    want = _expected(x, length, limited, mixed)
    # fp32 accumulation on both sides, in other orders: a value near a rounding boundary falls to the other side now
    # and then and moves by one step of its format, at most 2^-8 (bf16) or 2^-11 (fp16) of itself; the weights of a
    # row sum to at most 1, so the context moves by at most one step of its largest term, here within twice the
    # largest context value
    bound = 2 * (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)
    context, expected = (out - x["residual"]) / x["scale"], (want - x["residual"]) / x["scale"]
    assert float((context - expected).abs().max()) <= bound * float(expected.abs().max().clamp_min(1.0))


# d 256: one output part, 512 and 768: two, each finding its own columns; the first and the last hidden column
@pytest.mark.parametrize("dtype,value", [(torch.bfloat16, torch.inf), (torch.float16, torch.nan), (torch.float16, -torch.inf)])
@pytest.mark.parametrize("slots,k,d", [(1, 8, 256), (2, 4, 512), (1, 16, 768), (4, 4, 512)])
def test_a_cache_row_that_is_not_finite_reaches_the_rows_that_selected_it(dtype, value, slots, k, d):
    from relation_lm.kernels.relation_reduce import relation_mlp_rows

    length = 90
    x = _case(dtype, 2, length, slots, k, 128, d, seed=d + k)
    mixed = slots > 1

    def run(expanded):
        out = torch.empty_like(x["residual"])
        relation_mlp_rows(out, expanded, x["operand"], x["anchor"], x["partner"], x["score"], x["active"] if mixed else None,
                          x["slot_weight"] if mixed else None, x["scale"], x["wm"], x["w2"], x["b2"], x["nw"], x["nb"], 1e-5,
                          x["residual"], slots, length, False)
        assert_status_clear()
        return out

    before = run(x["expanded"])
    N, H = 2 * length, 4 * d
    seq = torch.arange(N, device="cuda")[:, None] // length
    used = torch.isfinite(x["score"])                                       # pairs with a weight
    if mixed:
        used &= x["active"][..., None]
    for column in (0, 65, H // 2 + 31, H - 1):
        for half, row in ((0, 0), (1, 41), (0, 77)):
            expanded = x["expanded"].clone()
            expanded[1, row, half * H + column] = value
            if half:
                hit = ((x["partner"].clamp(0, length - 1) == row) & used).flatten(1).any(1)
            else:
                hit = ((x["anchor"].clamp(0, length - 1) == row)[..., None] & used).flatten(1).any(1)
            hit &= (seq == 1).squeeze(1)
            out = run(expanded)
            assert bool(hit.any()) and bool(out[hit].isnan().all())
            assert torch.equal(out[~hit], before[~hit])


# The shapes of test_few_hidden_units_and_many_tiles with eight tiles or more for every cluster (74 of two CTAs, 33 of
# four): a tile's marks are read in its last stage, when the rows of tiles three ahead have been announced.
@pytest.mark.parametrize("value", (torch.inf, torch.nan))
@pytest.mark.parametrize("batch,slots,k,rdim,d,hidden", [
    (93, 4, 8, 64, 64, 256), (93, 4, 8, 64, 64, 384), (93, 2, 16, 128, 256, 256), (42, 4, 8, 128, 512, 512),
    (42, 4, 8, 64, 512, 768), (93, 4, 8, 64, 384, 256), (42, 4, 8, 128, 768, 512), (42, 4, 8, 64, 768, 768),
])
def test_anchors_that_are_not_finite_in_every_tile_of_a_cluster(value, batch, slots, k, rdim, d, hidden):
    from relation_lm.kernels.relation_reduce import relation_mlp_rows

    length = 53
    x = _case(torch.bfloat16, batch, length, slots, k, rdim, d, d + hidden, hidden)
    # a pair of tiles is eight rows: the first of each selects both of the rows that will not be finite
    x["anchor"][::8, :2] = torch.tensor([17, 40], device="cuda", dtype=torch.int32)
    x["active"][::8, :2] = True
    x["score"][::8, :2, 0] = 1.0

    def run(expanded):
        out = torch.empty_like(x["residual"])
        relation_mlp_rows(out, expanded, x["operand"], x["anchor"], x["partner"], x["score"], x["active"], x["slot_weight"], x["scale"],
                          x["wm"], x["w2"], x["b2"], x["nw"], x["nb"], 1e-5, x["residual"], slots, length, False)
        assert_status_clear()
        return out

    before = run(x["expanded"])
    assert bool(before.isfinite().all())
    anchor = x["anchor"].clamp(0, length - 1)
    used = torch.isfinite(x["score"]).any(-1) & x["active"]                  # [row, slot]: some pair has a weight
    for row, column in ((17, 0), (40, hidden - 1)):
        expanded = x["expanded"].clone()
        expanded[:, row, column] = value
        hit = ((anchor == row) & used).any(1)
        assert bool(hit[::8].all())
        out = run(expanded)
        assert bool(out[hit].isnan().all())
        assert torch.equal(out[~hit], before[~hit])


def test_new_output_without_residual_or_scale():
    from relation_lm.kernels.relation_reduce import relation_mlp_rows

    x = _case(torch.bfloat16, 2, 40, 1, 8, 128, 512, seed=9)
    out = torch.full_like(x["residual"], float("nan"))
    relation_mlp_rows(out, x["expanded"], x["operand"], x["anchor"], x["partner"], x["score"], None, None, None, x["wm"],
                      x["w2"], x["b2"], x["nw"], x["nb"], 1e-5, None, 1, 40, True)
    x["residual"].zero_()
    x["scale"].fill_(1.0)
    want = _expected(x, 40, True, False)
    assert float((out - want).abs().max()) <= 2 * 2 ** -8 * float(want.abs().max())
    assert_status_clear()


def test_sizes_outside_the_range_are_refused():
    from relation_lm.kernels.relation_reduce import relation_mlp_rows, relation_mlp_rows_supported

    assert not relation_mlp_rows_supported(6, 1, 128, 2048, 512, torch.bfloat16)
    assert not relation_mlp_rows_supported(2, 1, 128, 2048, 512, torch.bfloat16)
    assert not relation_mlp_rows_supported(8, 8, 128, 2048, 512, torch.bfloat16)
    assert not relation_mlp_rows_supported(8, 1, 128, 4096, 1024, torch.bfloat16)
    assert not relation_mlp_rows_supported(8, 1, 128, 2048, 512, torch.float32)
    x = _case(torch.bfloat16, 1, 8, 1, 6, 128, 128, seed=3)
    with pytest.raises(ValueError):
        relation_mlp_rows(x["residual"], x["expanded"], x["operand"], x["anchor"], x["partner"], x["score"], None, None, None,
                          x["wm"], x["w2"], x["b2"], x["nw"], x["nb"], 1e-5, None, 1, 8, True)
