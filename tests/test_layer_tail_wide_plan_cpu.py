"""Shared memory of the relation layer tail at d 768: what its warps use at the same time lies apart, inside the plan."""
from __future__ import annotations

import ctypes

import pytest

from relation_lm.kernels import _abi


@pytest.mark.parametrize("relation_dim,n_query", [(128, 256), (128, 0), (64, 0)])
@pytest.mark.parametrize("n_seq,k_out", [(1, 8), (2, 8), (8, 2), (4, 8), (8, 8), (1, 64)])
def test_buffers_of_the_kernels_end_are_disjoint(relation_dim, n_query, n_seq, k_out):
    ranges = (ctypes.c_int64 * 12)()
    assert _abi.LIB.rlm_selftest_layer_tail_plan(n_seq * k_out, n_seq, relation_dim, 768, n_query, ranges) == 0
    places = [(ranges[2 * i], ranges[2 * i + 1]) for i in range(5)]
    assert ranges[11] <= 232448 - 2048
    for begin, end in places:
        assert 0 <= begin <= end <= ranges[11]
    for i, (begin, end) in enumerate(places):
        for other_begin, other_end in places[:i]:
            assert end <= other_begin or other_end <= begin or begin == end or other_begin == other_end
