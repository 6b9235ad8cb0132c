"""The relation tail of a layer at d 768 (hidden slices shared by neighbouring CTAs, second-layer weights streamed) against
the oracle's unfused composition: every output within 1e-2 of its row's largest magnitude (16-bit operands, fp32
accumulation), two calls bit for bit the same."""
from __future__ import annotations

import pytest
import torch

import oracle
from gpu_util import assert_rel_close, assert_status_clear, position_tensor
from test_gpu_layer_tail import _case, _expected

pytestmark = pytest.mark.gpu


def _run(x, t, dtype):
    from relation_lm.kernels.relation_reduce import relation_layer_tail_wide

    dev = {k: (v.cuda() if isinstance(v, torch.Tensor) else v) for k, v in x.items()}
    B, d = x["hidden"].shape
    hidden = dev["hidden"].clone()
    normalized = torch.full((B, d), float("nan"), device="cuda", dtype=dtype)
    query = torch.full((B, x["wq"].size(0)), float("nan"), device="cuda", dtype=dtype) if x["wq"] is not None else None
    relation_layer_tail_wide(dev["expanded"], dev["operand"], dev["anchor"], dev["partner"], dev["scores"], dev["wm"],
                             dev["w2"], dev["b2"], dev["gamma"], dev["beta"], position_tensor(t), 1e-5, hidden,
                             dev["mix"], dev["next_w"], dev["next_b"], 1e-5, normalized, dev["wq"], query)
    return hidden, normalized, query


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,K,R,T,n_query,t", [
    (1, 8, 128, 64, 256, 3),          # 8 pairs in one cluster
    (2, 1, 128, 30, 256, 29),         # one pair a cluster
    (3, 5, 128, 40, 256, 39),         # fours of pairs that are not full
    (8, 8, 128, 96, 256, 95),         # 16 pairs a cluster
    (13, 8, 128, 50, 0, 20),          # 32 pairs, a last cluster with one sequence
    (25, 8, 128, 50, 256, 49),        # 56 pairs (seven sequences) a cluster
    (32, 2, 64, 30, 0, 10),           # relation width 64, eight sequences of two partners
    (64, 8, 128, 70, 256, 69),        # 64 pairs in each of eight clusters
    (1, 64, 128, 80, 256, 79),        # one sequence of 64 partners
])
def test_wide_tail_matches_unfused_oracle(B, K, R, T, n_query, t, dtype):
    from relation_lm.kernels.relation_reduce import relation_layer_tail_wide_supported

    assert relation_layer_tail_wide_supported(B, K, R, 3072, 768, n_query, dtype)
    x = _case(B, K, 768, R, T, n_query, dtype, 8100 + B)
    want_hidden, want_norm = _expected(x, t, dtype)
    hidden, normalized, query = _run(x, t, dtype)
    assert_rel_close(hidden, want_hidden, 1e-2, "residual")
    assert_rel_close(normalized, want_norm, 1e-2, "normalized")
    if n_query:
        assert_rel_close(query, oracle.linear(normalized.cpu(), x["wq"]), 1e-2, "query")
    for _ in range(20):
        again = _run(x, t, dtype)
        assert torch.equal(hidden, again[0]) and torch.equal(normalized, again[1])
        assert query is None or torch.equal(query, again[2])
    if B > 1:                               # the sequence without partners keeps its residual row
        assert torch.equal(hidden[1].cpu(), x["hidden"][1])
    assert_status_clear()


def test_wide_tail_rejects_other_widths():
    from relation_lm.kernels.relation_reduce import relation_layer_tail_wide_supported

    assert not relation_layer_tail_wide_supported(8, 8, 128, 2048, 512, 256, torch.bfloat16)
    assert not relation_layer_tail_wide_supported(8, 8, 256, 3072, 768, 256, torch.bfloat16)      # the ring does not fit
    with pytest.raises(ValueError):
        _run(_case(2, 8, 512, 128, 16, 0, torch.bfloat16, 1), 5, torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,K", [(1, 8), (4, 5), (8, 8), (28, 8), (56, 4)])
def test_wide_tail_is_no_further_from_64_bits_than_the_separate_kernels(B, K, dtype):
    """The separate launches that this tail stands for below 256 pairs keep the products of the operand rows in fp32 and
    the second layer's rows in 16 bits; the tail has all bits of the products, too, and its rows in fp32.  Both against
    the composition in 64 bits: residual rows and normalised rows, root mean square."""
    import torch.nn.functional as F

    from relation_lm.kernels.relation_reduce import relation_hidden_cached_out, relation_norm_reduce_residual_norm

    T, t, R = 96, 95, 128
    x = _case(B, K, 768, R, T, 256, dtype, 8600 + B)
    x["partner"], x["scores"] = x["partner"].clamp(min=0), torch.randn(B, K, generator=torch.Generator().manual_seed(B))
    hidden, normalized, _ = _run(x, t, dtype)

    dev = {k: (v.cuda() if isinstance(v, torch.Tensor) else v) for k, v in x.items()}
    rows = torch.empty(B, K, 3072, device="cuda", dtype=dtype)
    relation_hidden_cached_out(rows, dev["expanded"], dev["operand"], dev["anchor"], dev["partner"], dev["wm"])
    separate, separate_norm = dev["hidden"].clone(), torch.empty(B, 768, device="cuda", dtype=dtype)
    relation_norm_reduce_residual_norm(F.linear(rows, dev["w2"], dev["b2"]), dev["scores"], dev["gamma"], dev["beta"], position_tensor(t),
                                       1e-5, separate, dev["mix"], dev["next_w"], dev["next_b"], 1e-5, separate_norm)

    w = {k: (v.double() if v.is_floating_point() else v.long()) for k, v in dev.items() if isinstance(v, torch.Tensor)}
    seq = torch.arange(B, device="cuda")
    products = w["operand"][seq, w["anchor"]][:, None] * w["operand"][seq[:, None], w["partner"]]
    first = w["expanded"][seq, w["anchor"], :3072][:, None] + w["expanded"][seq[:, None], w["partner"], 3072:] + products @ w["wm"].T
    second = F.layer_norm(F.gelu(first) @ w["w2"].T + w["b2"], (768,), w["gamma"], w["beta"], 1e-5)
    active = torch.arange(K, device="cuda") < 7                                  # ceil(log2(t + 2)) partners take part
    weight = torch.softmax(w["scores"].masked_fill(~active, -torch.inf), 1)
    exact = w["hidden"] + w["mix"] * (weight[..., None] * second).sum(1)
    exact_norm = F.layer_norm(exact, (768,), w["next_w"], w["next_b"], 1e-5)
    off = lambda got, want: float((got.double() - want).square().mean().sqrt())  # noqa: E731
    assert off(hidden, exact) <= off(separate, exact)
    assert off(normalized, exact_norm) <= 1.02 * off(separate_norm, exact_norm)  # (both are its rounding to 16 bits)
    assert_status_clear()
