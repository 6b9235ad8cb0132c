"""The one-launch sequence state against column copies and ``router_cache_prefill`` over zeroed caches, bit for
bit, and the many-row LayerNorm cast against PyTorch's."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear

pytestmark = pytest.mark.gpu


def _by_parts(packed, slots, rdim, bs, wa, wp):
    from relation_lm.kernels.router_cache import router_cache_prefill

    B, T, _ = packed.shape
    n = max(slots, 1)
    at = (lambda s: 384 * s) if slots else (lambda s: 0)
    pa = 128 if slots else 128 + rdim
    cut = lambda s, lo, hi: packed[..., at(s) + lo:at(s) + hi]  # noqa: E731
    zeros = lambda *shape: torch.zeros(*shape, device="cuda", dtype=packed.dtype)  # noqa: E731
    want = {"anchor_keys": torch.stack([cut(s, 0, 64) for s in range(n)]),
            "partner_keys": torch.stack([cut(s, 64, 128) for s in range(n)]),
            "partner_anchor_cache": torch.stack([cut(s, pa, pa + 128) for s in range(n)]),
            "operand_cache": packed[..., 384 * slots:] if slots else packed[..., 128:128 + rdim]}
    caches = {k: zeros(n, B, T, 64) for k in ("anchor_raw_cache", "partner_raw_cache", "anchor_conv_cache", "partner_conv_cache")}
    stats = {k: zeros(n, B, T // bs, 4, 16) for k in ("anchor_mean", "anchor_std", "partner_mean", "partner_std")}
    for s in range(n):
        router_cache_prefill(cut(s, pa + 128, pa + 192), cut(s, pa + 192, pa + 256), *[c[s] for c in caches.values()],
                             *[c[s] for c in stats.values()], wa.view(n, 64, 3)[s], wp.view(n, 64, 3)[s], bs)
    want.update(caches, **stats)
    return {k: v if slots or k == "operand_cache" else v[0] for k, v in want.items()}


@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16))
@pytest.mark.parametrize("batch,blocks,bs,slots,rdim", [(1, 1, 1, 0, 128), (2, 3, 2, 0, 64), (1, 4, 8, 0, 128), (3, 5, 16, 2, 128),
                                                       (2, 2, 33, 1, 64), (2, 3, 64, 0, 128), (1, 2, 64, 4, 128), (1, 1, 256, 8, 8),
                                                       (1, 2, 451, 0, 64), (1, 2, 452, 0, 64), (2, 1, 600, 2, 128)])
def test_equals_copies_and_router_prefill(dtype, batch, blocks, bs, slots, rdim):
    from relation_lm.kernels.router_cache import STATE_NAMES, sequence_state

    g = torch.Generator(device="cuda").manual_seed(bs + 10 * slots)
    n = max(slots, 1)
    packed = torch.randn(batch, blocks * bs, 384 * n + rdim, generator=g, device="cuda").to(dtype)
    wa, wp = (torch.randn(n, 64, 3, generator=g, device="cuda") for _ in range(2))
    if not slots:
        wa, wp = wa[0], wp[0]
    got = sequence_state(packed, slots, rdim, bs, wa, wp)
    want = _by_parts(packed, slots, rdim, bs, wa, wp)
    for name in STATE_NAMES:
        assert got[name].shape == want[name].shape and torch.equal(got[name], want[name].contiguous()), name
    assert_status_clear()


def test_rejects_partial_blocks_and_other_dtypes():
    from relation_lm.kernels.router_cache import sequence_state

    w = torch.zeros(64, 3, device="cuda")
    with pytest.raises(ValueError):
        sequence_state(torch.zeros(1, 10, 512, device="cuda", dtype=torch.bfloat16), 0, 128, 4, w, w)
    with pytest.raises(ValueError):
        sequence_state(torch.zeros(1, 8, 512, device="cuda"), 0, 128, 4, w, w)


# widths at the edges of a lane's chunks, rows below and beyond one pass of the grid
@pytest.mark.parametrize("rows,d", [(1, 8), (3, 256), (5, 264), (17, 512), (9, 576), (20_000, 768), (7, 1024)])
def test_layer_norm_cast(rows, d):
    from relation_lm.kernels.packed_projection import layer_norm_cast

    g = torch.Generator(device="cuda").manual_seed(d)
    x = torch.randn(rows, d, generator=g, device="cuda") * 3 + 1
    gamma, beta = torch.randn(d, generator=g, device="cuda"), torch.randn(d, generator=g, device="cuda")
    for dtype, step in ((torch.bfloat16, 2 ** -8), (torch.float16, 2 ** -11)):
        out = torch.empty(rows, d, device="cuda", dtype=dtype)
        layer_norm_cast(x, gamma, beta, 1e-5, out)
        want = torch.nn.functional.layer_norm(x, (d,), gamma, beta, 1e-5)
        # one rounding to the output's format, plus fp32 sums in another order (d 1024 terms: below 1e-5 of a value)
        assert bool(((out.float() - want).abs() <= (step + 1e-5) * want.abs() + 1e-5).all())
