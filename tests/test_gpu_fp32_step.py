"""Single-precision outputs of the kernels that carry a LayerNorm for the next one, against float64."""
from __future__ import annotations

import pytest
import torch

from gpu_util import assert_status_clear, position_tensor

pytestmark = pytest.mark.gpu

# A normalised value is (x - mean) * rstd * w + b with |x - mean| * rstd <= sqrt(d) <= 32.  The sums of the mean and the
# variance are trees of depth <= log2(1024) + 2, each level one rounding of 2^-24: 12 * 6e-8 relative on either, and
# four roundings more for the value itself, 16 * 6e-8 * 32 < 4e-5 for the largest value and in proportion below.
BOUND = 16 * 2.0 ** -24


def _close(got, want, scale):
    err = (got.double() - want).abs()
    assert bool((err <= BOUND * (scale + 1.0)).all()), float((err / (scale + 1.0)).max())


@pytest.mark.parametrize("B,d", [(1, 8), (3, 260), (2, 1024)])
def test_embedding_with_fp32_layer_norms(B, d):
    from relation_lm.kernels.packed_projection import decode_embed_norm

    g = torch.Generator(device="cuda").manual_seed(d)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    tok, bnd, pos, w1, b1, w2, b2 = r(50, d), r(7, d), r(9, d), r(d), r(d), r(d), r(d)
    tokens, bounds = torch.randint(0, 50, (B,), device="cuda"), torch.randint(0, 7, (B,), device="cuda")
    n1, n2 = torch.empty(B, d, device="cuda"), torch.empty(B, d, device="cuda")
    out = decode_embed_norm(tokens, bounds, tok, bnd, pos, position_tensor(5), 1.5, w1, b1, n1, w2, b2, n2, 1e-5)
    x = (tok[tokens] + bnd[bounds]) * 1.5 + pos[5]
    assert torch.allclose(out, x, rtol=2.0 ** -22, atol=2.0 ** -22)       # one fused multiply-add or two roundings
    for got, w, b in ((n1, w1, b1), (n2, w2, b2)):
        want = torch.nn.functional.layer_norm(out.double(), (d,), w.double(), b.double(), 1e-5)
        _close(got, want, ((want - b.double()).abs().amax(-1, keepdim=True)) + b.abs().double())
    assert_status_clear()


@pytest.mark.parametrize("B,K,D", [(1, 1, 8), (3, 8, 264), (2, 9, 1024)])
def test_norm_reduce_with_an_fp32_next_layer_norm(B, K, D):
    from relation_lm.kernels.relation_reduce import relation_norm_reduce, relation_norm_reduce_residual_norm

    g = torch.Generator(device="cuda").manual_seed(D)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    raw, scores, gamma, beta, hidden, w, b = r(B, K, D), r(B, K), r(D), r(D), r(B, D), r(D), r(D)
    mix, before, normalized = torch.tensor([0.3], device="cuda"), hidden.clone(), torch.empty(B, D, device="cuda")
    context = relation_norm_reduce(raw, scores, gamma, beta, position_tensor(600), 1e-5)
    relation_norm_reduce_residual_norm(raw, scores, gamma, beta, position_tensor(600), 1e-5, hidden, mix, w, b, 1e-5,
                                       normalized)
    assert torch.allclose(hidden, before + 0.3 * context, rtol=2.0 ** -22, atol=2.0 ** -21)
    want = torch.nn.functional.layer_norm(hidden.double(), (D,), w.double(), b.double(), 1e-5)
    _close(normalized, want, ((want - b.double()).abs().amax(-1, keepdim=True)) + b.abs().double())
    assert_status_clear()
