"""Whole-sequence selectors at each tile size (one, two or four positions per warp, chosen by the number of
tiles against the SMs) and 16-bit dtype, against the per-row kernels bit for bit."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear

pytestmark = pytest.mark.gpu

T, NB, L, TOP = 250, 10, 32, 2     # blocks of 25: a ragged tile at every size, no power of two


def _inputs(B, slots, dtype):
    g = torch.Generator(device="cuda").manual_seed(77 + B)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    N, lead, mid = B * T, (slots,) if slots else (), (slots,) if slots else ()
    return [r(N, *mid, 64).to(dtype), r(*lead, B, T, 64).to(dtype), r(N, *mid, 64).to(dtype),
            r(*lead, B, NB, 4, 16).to(dtype), r(*lead, B, NB, 4, 16).abs().to(dtype), r(*lead, 4), r(*lead, 4, 16),
            r(N, *mid, 128).to(dtype), r(*lead, B, T, 128).to(dtype), r(*lead, B, T, 64).to(dtype),
            r(*lead, B, NB, 4, 16).to(dtype), r(*lead, B, NB, 4, 16).abs().to(dtype), r(*lead, 4), r(*lead, 4, 16)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("slots", [0, 3])
@pytest.mark.parametrize("B", [2, 8, 13, 37, 74])     # 8, 16 and 24 warps of a position, 32 of two and of four
def test_tiled_selector_equals_the_per_row_selector(B, slots, dtype):
    from relation_lm.kernels.multi_select import relation_select_multi_prefill, relation_select_multi_rows
    from relation_lm.kernels.relation_select import relation_select_packed_prefill, relation_select_packed_rows

    x = _inputs(B, slots, dtype)
    row_batch = torch.arange(B, dtype=torch.int32, device="cuda").repeat_interleave(T)
    row_pos = torch.arange(T, dtype=torch.int32, device="cuda").repeat(B)
    tiled, rows = (relation_select_multi_prefill, relation_select_multi_rows) if slots else \
        (relation_select_packed_prefill, relation_select_packed_rows)
    got = tiled(*x, T, L, TOP, 4, False)
    want = rows(*x, row_batch, row_pos, L, TOP, 4, False)
    for mine, theirs in zip(got, want):
        assert torch.equal(mine.view(torch.int32) if mine.dtype == torch.float32 else mine,
                           theirs.view(torch.int32) if theirs.dtype == torch.float32 else theirs)
    assert_status_clear()


@pytest.mark.parametrize("T,NB,L,top", [(256, 4, 24, 3),     # blocks of 64, a window that is no multiple of 32
                                        (512, 128, 32, 4),   # 128 blocks of 4: eight to a pass
                                        (320, 10, 100, 1),   # blocks of 32: one to a pass
                                        (96, 3, 17, 0)])     # no remote blocks
@pytest.mark.parametrize("strict", [False, True])
def test_pass_shapes_of_the_tiled_selector(T, NB, L, top, strict):
    """Ragged windows and every relation of the block size to a pass of 32 rows."""
    from relation_lm.kernels.relation_select import relation_select_packed_prefill, relation_select_packed_rows

    B, dtype = 2, torch.float16
    g = torch.Generator(device="cuda").manual_seed(5 * T + top)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    stats = lambda: (r(B, NB, 4, 16).to(dtype), r(B, NB, 4, 16).abs().to(dtype), r(4), r(4, 16))  # noqa: E731
    x = [r(B * T, 64).to(dtype), r(B, T, 64).to(dtype), r(B * T, 64).to(dtype), *stats(), r(B * T, 128).to(dtype),
         r(B, T, 128).to(dtype), r(B, T, 64).to(dtype), *stats()]
    row_batch = torch.arange(B, dtype=torch.int32, device="cuda").repeat_interleave(T)
    row_pos = torch.arange(T, dtype=torch.int32, device="cuda").repeat(B)
    got = relation_select_packed_prefill(*x, T, L, top, 8, strict)
    want = relation_select_packed_rows(*x, row_batch, row_pos, L, top, 8, strict)
    for mine, theirs in zip(got, want):
        assert torch.equal(mine.view(torch.int32), theirs.view(torch.int32))
    assert_status_clear()
