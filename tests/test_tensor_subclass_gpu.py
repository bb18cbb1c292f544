"""Tensor subclasses without a dispatch of their own keep their type through the operators that allocate like their operands."""

import pytest
import torch

import oops_b200 as oops

pytestmark = pytest.mark.gpu


class Labelled(torch.Tensor):
    pass


def label(t):
    return t.as_subclass(Labelled)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_results_keep_the_type(cuda, dtype):
    q = torch.randn(1, 5, 24, 2, 32, device=cuda, dtype=dtype, requires_grad=True)
    tokens = torch.randn(2, 3, 16, 24, device=cuda, dtype=dtype, requires_grad=True)
    values, single = torch.randn(2, 2, 8, 16, device=cuda, dtype=dtype), torch.randn(2, 8, 24, device=cuda, dtype=dtype)
    weights = torch.randn(32, 24, device=cuda, dtype=dtype), torch.randn(24, 32, device=cuda, dtype=dtype)
    for call, leaf in ((lambda t: oops.triangle_attention(t, t, t), q), (lambda t: oops.pair_bias_attention(t, t, t), tokens),
                       (lambda t: oops.gate_attention_output(values, t, *weights), single.requires_grad_(True))):
        want = call(leaf)
        got = call(label(leaf))
        assert type(got) is Labelled and torch.equal(got.as_subclass(torch.Tensor), want)
        first, second = (torch.autograd.grad(out.as_subclass(torch.Tensor).sum(), leaf)[0].as_subclass(torch.Tensor) for out in (got, want))
        # (the gradients of a tensor that is query, key and value at once are added in the order the engine meets them)
        assert float((first - second).norm()) <= 4 * torch.finfo(dtype).eps * float(second.norm())
    parameter = torch.nn.Parameter(q.detach())
    assert type(oops.triangle_attention(parameter, parameter, parameter)) is torch.Tensor
