"""What surrounds the operators in PyTorch's dispatcher, on fake CUDA tensors: version counters, gradients, transforms."""
from __future__ import annotations

import pytest
import torch
import torch.autograd.forward_ad as forward_ad
from torch._subclasses.fake_tensor import FakeTensorMode

from relation_lm.kernels import relation_reduce as rr
from relation_lm.kernels.packed_projection import greedy_token


@pytest.fixture(autouse=True)
def fake_cuda():
    with FakeTensorMode():
        yield


def zeros(*shape, dtype=torch.float32):
    return torch.zeros(*shape, device="cuda", dtype=dtype)


def parameter(*shape):
    return torch.nn.Parameter(zeros(*shape))


def reduce(raw=None, weight=None):
    return rr.relation_norm_reduce(zeros(1, 8, 16) if raw is None else raw, zeros(1, 8), zeros(16) if weight is None else weight,
                                   zeros(16), zeros(1, dtype=torch.int64), 1e-5)


def reduce_into(hidden, weight=None):
    rr.relation_norm_reduce_residual(zeros(1, 8, 16), zeros(1, 8), zeros(16) if weight is None else weight, zeros(16),
                                     zeros(1, dtype=torch.int64), 1e-5, hidden, zeros(1))


def update(expanded, weights):
    index = zeros(1, 2, dtype=torch.int32)
    return rr.relation_hidden_cache_update(expanded, zeros(1, 4, 8), index[:, 0].contiguous(), index, *weights,
                                           zeros(1, dtype=torch.int64))


def test_version_counters_of_written_arguments_advance():
    hidden = zeros(1, 16)
    reduce_into(hidden)
    assert hidden._version == 1
    with torch.no_grad():
        reduce_into(hidden)
    assert hidden._version == 2
    expanded = zeros(1, 4, 32)
    update(expanded, [zeros(16, 8), zeros(16, 8), zeros(16, 8), zeros(16)])
    assert expanded._version == 1
    position, logits = zeros(1, dtype=torch.int64), zeros(2, 8)
    greedy_token(logits, 8, position)
    assert position._version == 1 and logits._version == 0


def test_results_of_parameters_ask_for_a_derivative_that_does_not_exist():
    out = reduce(weight=parameter(16))
    assert out.requires_grad and out.grad_fn is not None
    with torch.no_grad():
        assert not reduce(weight=parameter(16)).requires_grad
    assert not reduce().requires_grad
    expanded = zeros(1, 4, 32)
    assert update(expanded, [parameter(16, 8), parameter(16, 8), parameter(16, 8), parameter(16)]).requires_grad
    assert not expanded.requires_grad           # what is written is left alone
    assert not greedy_token(zeros(2, 8).requires_grad_(), 8).requires_grad      # whole numbers


def test_leaves_that_require_a_derivative_may_be_written():
    hidden = parameter(1, 16)
    reduce_into(hidden)
    assert hidden.is_leaf and hidden._version == 1
    reduce_into(parameter(2, 1, 16)[0])         # a view of one
    reduce_into(zeros(1, 16), weight=parameter(16))


def test_transforms():
    assert torch.vmap(reduce)(zeros(3, 1, 8, 16)).shape == (3, 1, 16)
    with forward_ad.dual_level():
        out = reduce(forward_ad.make_dual(zeros(1, 8, 16), zeros(1, 8, 16)))
        assert forward_ad.unpack_dual(out).tangent is None
