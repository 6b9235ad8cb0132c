"""The selectors of warp passes: whole-sequence forms at each tile size (one, two or four
positions per warp, chosen by the number of tiles against the SMs) and the decode form, in either 16-bit dtype,
against the per-row kernels bit for bit."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear, position_tensor

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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,NB,L,top,K,positions", [
    (128, 8, 17, 2, 8, (0, 15, 16, 127)),            # resident caches, ragged window, no complete block at first
    (2048, 32, 128, 2, 8, (63, 1000, 2047)),         # picked rows from L2
    (600, 150, 40, 5, 4, (3, 300, 599)),             # more than 128 blocks, blocks of 4, passes of several blocks
    (1024, 16, 400, 3, 8, (500, 1023)),              # more than 512 candidates: the block-wide top-K
    (320, 5, 33, 0, 8, (0, 32, 319)),                # no remote blocks
])
def test_decode_form_equals_the_rows_form(T, NB, L, top, K, positions, dtype):
    from relation_lm.kernels.relation_select import relation_select_packed, relation_select_packed_rows

    B = 3
    g = torch.Generator(device="cuda").manual_seed(T + L)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    stats = lambda: (r(B, NB, 4, 16).to(dtype), r(B, NB, 4, 16).abs().to(dtype), r(4), r(4, 16))  # noqa: E731
    x = [r(B, 64).to(dtype), r(B, T, 64).to(dtype), r(B, 64).to(dtype), *stats(), r(B, 128).to(dtype),
         r(B, T, 128).to(dtype), r(B, T, 64).to(dtype), *stats()]
    x[1][:, 5] = x[1][:, 3]                          # equal keys: the lower position wins
    x[9][:, 5] = x[9][:, 3]
    row_batch = torch.arange(B, dtype=torch.int32, device="cuda")
    for t in positions:
        got = relation_select_packed(*x, position_tensor(t), L, top, K, False)
        want = relation_select_packed_rows(*x, row_batch, torch.full_like(row_batch, t), L, top, K, False)
        for mine, theirs in zip(got, want):
            assert torch.equal(mine.view(torch.int32), theirs.view(torch.int32)), t
    assert_status_clear()
