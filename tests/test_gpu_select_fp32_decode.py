"""Decode launches of the selector in single precision (a warp pass per phase, whole key caches staged where they
fit) against the per-row form of the same queries, and against the oracle where caches hold values that are not
finite: indices and scores bit for bit."""
from __future__ import annotations

import pytest
import torch

import cases
import oracle
from gpu_util import assert_status_clear, position_tensor, select_args, to_cuda

pytestmark = pytest.mark.gpu


def _equal(a, b):
    if a.dtype != torch.float32:
        return torch.equal(a, b)
    nan = a.isnan()
    return torch.equal(nan, b.isnan()) and torch.equal(a[~nan].view(torch.int32), b[~nan].view(torch.int32))


SHAPES = [
    (1, 128, 8, 32, 2, 8),        # both key caches staged
    (5, 352, 11, 48, 3, 4),       # ... close to the largest context that fits, 11 blocks of 32
    (2, 512, 64, 16, 2, 8),       # window staged, blocks of 8 read where they lie
    (3, 120, 40, 7, 4, 5),        # blocks of 3: passes that cross blocks
    (2, 300, 150, 20, 8, 16),     # more than 128 blocks
    (2, 1024, 16, 64, 0, 8),      # no remote blocks
    (2, 1024, 16, 64, 4, 32),     # 320 candidates
    (1, 2048, 16, 40, 4, 8),      # 552 candidates
    (297, 64, 8, 16, 2, 8),       # more rows than two per SM: the general form
    (2, 384, 12, 32, 2, 8),       # both key caches staged, blocks of 32
    (2, 416, 13, 32, 2, 8),       # ... a block more: the window
    (2, 344, 43, 16, 2, 8),       # both staged, blocks of 8
    (2, 352, 44, 16, 2, 8),       # ... a block more: the window
    (149, 352, 11, 64, 8, 8),     # two rows an SM, more picked rows than a pass per warp
    (2, 512, 64, 16, 4, 8),       # the most short blocks this form chooses
    (2, 512, 64, 16, 5, 8),       # ... and one more: the general form
]


def _case(B, T, NB, L, top, K):
    return {"kind": "select", "seed": 7400 + T + K, "batch": B, "context": T, "blocks": NB, "local_window": L,
            "top_blocks": top, "k_out": K, "strict_valid": False, "dtype": "fp32"}


def _positions(T, NB, L):
    bs = T // NB
    return sorted({0, 1, L - 1, L, bs, 2 * bs + 1, T // 2, T - 2, T - 1} & set(range(T)))


@pytest.mark.parametrize("B,T,NB,L,top,K", SHAPES)
def test_decode_form_equals_the_rows_form(B, T, NB, L, top, K):
    from relation_lm.kernels.relation_select import relation_select_packed, relation_select_packed_rows

    args = select_args(to_cuda(cases.make_inputs(_case(B, T, NB, L, top, K))))
    rows = torch.arange(B, dtype=torch.int32).cuda()
    for strict in (False, True):
        for t in _positions(T, NB, L):
            got = relation_select_packed(*args, position_tensor(t), L, top, K, strict)
            ref = relation_select_packed_rows(*args, rows, torch.full_like(rows, t), L, top, K, strict)
            for a, b in zip(got, ref):
                assert _equal(a, b), (t, strict)
    assert_status_clear()


@pytest.mark.parametrize("B,T,NB,L,top,K", SHAPES[:5])
def test_caches_with_values_that_are_not_finite(B, T, NB, L, top, K):
    """Key rows that score +-inf (ties go to the lowest position), rows of zeros, an infinite block statistic."""
    from relation_lm.kernels.relation_select import relation_select_packed

    args = [x.clone() for x in select_args(cases.make_inputs(_case(B, T, NB, L, top, K)))]
    for i in (1, 9):
        args[i][:, 3::17, 5] = float("inf")
        args[i][:, 11::31] = 0.0
    args[3].view(B, NB, -1)[:, 1::5, 9] = float("-inf")
    on_gpu = [x.cuda() for x in args]
    for t in _positions(T, NB, L):
        got = relation_select_packed(*on_gpu, position_tensor(t), L, top, K, False)
        want = oracle.relation_select(*args, t, L, top, K, False)
        for a, b in zip(got, want):
            assert _equal(a.cpu(), b), t
    assert_status_clear()


# blocks a lane each, four a lane, blocks ranked against one another; up to 256 candidates, 320 and 552
@pytest.mark.parametrize("B,T,NB,L,top,K", [SHAPES[i] for i in (0, 2, 3, 4, 6, 7)])
@pytest.mark.parametrize("where", ["statistics", "keys", "both"])
def test_scores_that_are_nan_rank_as_in_the_rows_form(B, T, NB, L, top, K, where):
    from relation_lm.kernels.relation_select import relation_select_packed, relation_select_packed_rows

    args = [x.clone() for x in select_args(to_cuda(cases.make_inputs(_case(B, T, NB, L, top, K))))]
    for i in (1, 9):
        if where != "statistics":
            args[i][:, 5::37, 5] = float("nan")
    for i in (3, 10):
        if where != "keys":
            args[i].view(B, NB, -1)[:, 2::7] = float("nan")
    rows = torch.arange(B, dtype=torch.int32).cuda()
    for t in _positions(T, NB, L):
        got = relation_select_packed(*args, position_tensor(t), L, top, K, False)
        ref = relation_select_packed_rows(*args, rows, torch.full_like(rows, t), L, top, K, False)
        for a, b in zip(got, ref):
            assert _equal(a, b), t
    assert_status_clear()


def test_strided_queries_and_query_views_off_16_bytes():
    """Queries as columns of one matrix whose rows start anywhere, as a step hands them over."""
    from relation_lm.kernels.relation_select import relation_select_packed

    case = {"kind": "select", "seed": 7451, "batch": 3, "context": 128, "blocks": 8, "local_window": 32,
            "top_blocks": 2, "k_out": 8, "strict_valid": False, "dtype": "fp32"}
    args = list(select_args(to_cuda(cases.make_inputs(case))))
    want = relation_select_packed(*args, position_tensor(100), 32, 2, 8, False)
    wide = torch.zeros(3, 259, device="cuda")
    at = {0: slice(1, 65), 2: slice(65, 129), 7: slice(129, 257)}
    for i, columns in at.items():
        wide[:, columns] = args[i]
        args[i] = wide[:, columns]
    got = relation_select_packed(*args, position_tensor(100), 32, 2, 8, False)
    assert all(_equal(a, b) for a, b in zip(got, want))
    assert_status_clear()
