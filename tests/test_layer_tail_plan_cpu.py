"""Shared memory of the relation layer tail: what its warps use at the same time lies apart."""
from __future__ import annotations

import ctypes

import pytest

from relation_lm.kernels import _abi

NAMES = ("normalised pairs", "16-bit rows", "residual rows", "statistics", "query weights")


@pytest.mark.parametrize("d_model,relation_dim,n_query", [(512, 128, 256), (512, 64, 0), (256, 128, 256), (128, 64, 128)])
@pytest.mark.parametrize("n_seq,k_out", [(1, 8), (1, 1), (2, 8), (4, 8), (8, 8), (8, 4), (1, 64)])
def test_buffers_of_the_kernels_end_are_disjoint(d_model, relation_dim, n_query, n_seq, k_out):
    """A warp may be at its last LayerNorm while another of its CTA still sums its normalised pairs, pushes residual
    columns or reads the query weights: no two of these places may share a byte, and all lie inside the plan."""
    ranges = (ctypes.c_int64 * 12)()
    assert _abi.LIB.rlm_selftest_layer_tail_plan(n_seq * k_out, n_seq, relation_dim, d_model, n_query, ranges) == 0
    places = [(ranges[2 * i], ranges[2 * i + 1], NAMES[i]) for i in range(5)]
    for begin, end, name in places:
        assert 0 <= begin <= end <= ranges[11], name
    for i, (begin, end, name) in enumerate(places):
        for other_begin, other_end, other in places[:i]:
            assert end <= other_begin or other_end <= begin or begin == end or other_begin == other_end, (name, other)
