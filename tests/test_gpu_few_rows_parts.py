"""Single-precision products of several passes of rows, the passes on CTAs of their own or in one CTA: on both sides of
the rules' lines (columns that fill two CTAs an SM, waves against passes, eight or sixteen rows a pass), against 64-bit
products, and each row the same bits as alone with seven others."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [9, 16, 17, 24, 33, 64])
@pytest.mark.parametrize("d_in,n_out", [(2048, 592), (2044, 600), (1024, 1184), (1024, 1185), (2304, 576), (1920, 40), (1536, 768)])
def test_passes(rows, d_in, n_out):
    from relation_lm.kernels.packed_projection import few_rows_projection

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n_out = n_out * sms // 148                     # (the lines lie at multiples of the SM count)
    g = torch.Generator().manual_seed(100 * rows + d_in + n_out)
    x, w = torch.randn(rows, d_in, generator=g).cuda(), torch.randn(n_out, d_in, generator=g).cuda()
    b, room = torch.randn(n_out, generator=g).cuda(), torch.full((rows * n_out + 64,), 7.0, device="cuda")
    out = room[:rows * n_out].view(rows, n_out)
    few_rows_projection(out, x, w, b)
    # at most d_in / 32 roundings in a lane's chain, ten over lanes and warps
    bound = (d_in / 32 + 10) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + b.double().abs())
    assert bool(((out.double() - (x.double() @ w.double().T + b.double())).abs() <= bound).all())
    assert bool((room[rows * n_out:] == 7.0).all())
    last = torch.empty(8, n_out, device="cuda")
    few_rows_projection(last, x[-8:], w, b)
    assert torch.equal(last, out[-8:])
    assert_status_clear()
