"""Whole-sequence anchor scores from queries kept in 16 bits, at the ends of the type's range: subnormal keys, block
statistics and queries, signed zeros, large values, infinities (no score is NaN: where one is, the forms rank it
apart).  The per-row form widens every operand first; indices and scores agree bit for bit."""
from __future__ import annotations

import pytest
import torch

import cases
from gpu_util import assert_status_clear, select_args, to_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tiny", [("bf16", 2.0 ** -128), ("fp16", 2.0 ** -18)])
@pytest.mark.parametrize("T,NB,L", [(160, 10, 24), (96, 4, 70), (130, 26, 9)])
def test_extremes_equal_the_rows_form(dtype, tiny, T, NB, L):
    from relation_lm.kernels.relation_select import relation_select_packed_prefill, relation_select_packed_rows

    B, top, K = 2, 2, 4
    case = {"kind": "select", "seed": 7500 + T, "batch": B, "rows": B * T, "context": T, "blocks": NB, "local_window": L,
            "top_blocks": top, "k_out": K, "strict_valid": False, "dtype": dtype}
    args = [x.clone() for x in select_args(to_cuda(cases.make_inputs(case)))]
    keys, queries, mean = args[1], args[0], args[3].view(B, NB, 64)
    keys[:, 1::3] *= tiny                          # subnormal rows
    keys[:, 2::7, ::2] = -0.0
    keys[:, 4::11] *= 2.0 ** 6
    keys[1, 5::13, 7] = float("inf")
    queries[::5] *= tiny
    queries[1::17, 3] *= 2.0 ** 10
    args[2][3::9] *= tiny
    mean[:, 1::3] *= tiny
    rows = torch.arange(B, dtype=torch.int32).repeat_interleave(T).cuda()
    positions = torch.arange(T, dtype=torch.int32).repeat(B).cuda()
    got = relation_select_packed_prefill(*args, T, L, top, K, False)
    want = relation_select_packed_rows(*args, rows, positions, L, top, K, False)
    for a, b in zip(got, want):
        if a.dtype == torch.float32:
            nan = a.isnan()
            assert torch.equal(nan, b.isnan()) and torch.equal(a[~nan].view(torch.int32), b[~nan].view(torch.int32))
        else:
            assert torch.equal(a, b)
    assert_status_clear()
