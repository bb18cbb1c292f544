"""Gradients that have a graph: what the operators around the attention kernels give for a second differentiation is what their
composition from single operations gives, through every node that has a graph itself (the library's own nodes stop there).
Bound: f32 sums in another order, 2^-16 of the 2-norm."""

import pytest
import torch
from torch.nn import functional as F

import oops_b200 as oops
from oops_b200.runtime.native import native
from test_triangle_multiplication_gpu import _weights

pytestmark = pytest.mark.gpu


def second(f, leaves):
    out = f(*leaves)
    first = torch.autograd.grad(out, leaves, torch.ones_like(out), create_graph=True)
    graph = [g.requires_grad for g in first]
    total = sum((g.double() ** 2).sum() for g in first if g.requires_grad)
    return graph, [g.detach() for g in first], torch.autograd.grad(total, leaves, allow_unused=True)


def compare(operator, composed, values):
    results = [second(f, [v.detach().requires_grad_(True) for v in values]) for f in (operator, composed)]
    assert results[0][0] == results[1][0] and any(results[0][0])
    for got, want in zip((*results[0][1], *results[0][2]), (*results[1][1], *results[1][2])):
        assert (got is None) == (want is None)
        if got is not None:
            assert float((got - want).norm()) <= 2.0**-16 * float(want.norm()) + 1e-12


def test_gate_output(cuda):
    gen = torch.Generator().manual_seed(2)
    values = [torch.randn(*s, generator=gen).to(cuda) for s in ((2, 2, 8, 16), (2, 8, 24), (32, 24), (24, 32))]

    def composed(attention, single, gate_weight, output_weight):
        return F.linear(native().sigmoid_gate(attention, F.linear(single, gate_weight)), output_weight)

    compare(oops.gate_attention_output, composed, values)


@pytest.mark.parametrize("direction", ["outgoing", "incoming"])
@pytest.mark.parametrize("masked", [False, True])
def test_pair_update(cuda, direction, masked):
    gen = torch.Generator().manual_seed(3)
    weights = _weights(gen, 16, 24, masked)
    pair = torch.randn(2, 12, 12, 16, generator=gen).to(cuda)
    mask = torch.rand(2, 12, 12, generator=gen).to(cuda) if masked else None

    def operator(pair, *values):
        return oops.triangle_multiplication(pair, mask, direction=direction, **dict(zip(weights, values)))

    def composed(pair, *values):
        w = dict(zip(weights, values))
        x = oops.layer_norm(pair, 16, w["input_norm_weight"], w["input_norm_bias"])
        keep = 1.0 if mask is None else mask.unsqueeze(-1)
        left, right = (keep * torch.sigmoid(F.linear(x, w[f"{s}_gate_weight"], w.get(f"{s}_gate_bias")))
                       * F.linear(x, w[f"{s}_value_weight"], w.get(f"{s}_value_bias")) for s in ("left", "right"))
        update = torch.einsum("bikh,bjkh->bijh" if direction == "outgoing" else "bkih,bkjh->bijh", left, right).contiguous()
        normed = oops.layer_norm(update, 24, w["output_norm_weight"], w["output_norm_bias"])
        return F.linear(normed, w["output_weight"], w.get("output_bias")) * torch.sigmoid(F.linear(x, w["output_gate_weight"], w.get("output_gate_bias")))

    compare(operator, composed, [pair, *(w.to(cuda) for w in weights.values())])
