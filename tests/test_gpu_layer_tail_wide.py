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
