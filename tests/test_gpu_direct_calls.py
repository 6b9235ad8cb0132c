"""Operators called without the dispatcher: same results and checks, and the dispatcher wherever it has work to do."""
from __future__ import annotations

import pytest
import torch

from gpu_util import position_tensor

pytestmark = pytest.mark.gpu


def _reduce_args(device="cuda"):
    g = torch.Generator().manual_seed(3)
    raw, scores = torch.randn(2, 4, 64, generator=g).to(device), torch.randn(2, 4, generator=g).to(device)
    return raw, scores, torch.ones(64, device=device), torch.zeros(64, device=device), position_tensor(9), 1e-5


def test_same_result_as_the_dispatched_operator():
    from relation_lm.kernels.relation_reduce import relation_norm_reduce

    args = _reduce_args()
    assert torch.equal(relation_norm_reduce(*args), torch.ops.relation_lm.relation_norm_reduce.default(*args))


def test_written_arguments_advance_their_version():
    from relation_lm.kernels.packed_projection import layer_norm_cast

    out = torch.empty(4, 64, device="cuda")
    before = out._version
    layer_norm_cast(torch.randn(4, 64, device="cuda"), torch.ones(64, device="cuda"), torch.zeros(64, device="cuda"), 1e-5, out)
    assert out._version == before + 1


def test_errors_and_derivatives_are_the_dispatched_operators():
    from relation_lm.kernels.relation_reduce import relation_norm_reduce

    args = _reduce_args()
    with pytest.raises(ValueError):
        relation_norm_reduce(args[0], args[1][:, :3], *args[2:])            # shapes that do not agree
    with pytest.raises(NotImplementedError):
        relation_norm_reduce(*[a.cpu() if isinstance(a, torch.Tensor) else a for a in args])
    raw = args[0].clone().requires_grad_()
    out = relation_norm_reduce(raw, *args[1:])
    with pytest.raises(RuntimeError):
        out.sum().backward()


def test_modes_see_the_operator():
    from torch.utils._python_dispatch import TorchDispatchMode

    from relation_lm.kernels.relation_reduce import relation_norm_reduce

    seen = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Watch():
        relation_norm_reduce(*_reduce_args())
    assert any("relation_norm_reduce" in name for name in seen)


@pytest.mark.parametrize("direct", [True, False])
def test_a_saved_tensor_that_an_operator_overwrites_is_noticed(direct):
    """By an operator that is called directly and by one that goes through the dispatcher."""
    from relation_lm.kernels.relation_reduce import relation_norm_reduce_residual, relation_norm_reduce_residual_norm

    raw, scores, weight, bias, position, eps = _reduce_args()
    hidden, x = torch.randn(2, 64, device="cuda"), torch.ones(2, 64, device="cuda", requires_grad=True)
    y, mix = (x * hidden).sum(), torch.ones((), device="cuda")          # keeps `hidden` for the backward pass
    if direct:
        relation_norm_reduce_residual_norm(raw, scores, weight, bias, position, eps, hidden, mix, weight, bias, eps, torch.empty_like(hidden))
    else:
        relation_norm_reduce_residual(raw, scores, weight, bias, position, eps, hidden, mix)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward()


def test_views_that_are_still_to_be_negated():
    """The imaginary part of a conjugate is a view with a sign that the dispatcher resolves before the kernel."""
    from relation_lm.kernels.relation_reduce import relation_norm_reduce

    args = _reduce_args()
    lazy = torch._neg_view(args[1])
    assert lazy.is_neg()
    assert torch.equal(relation_norm_reduce(args[0], lazy, *args[2:]), relation_norm_reduce(args[0], lazy.resolve_neg(), *args[2:]))
