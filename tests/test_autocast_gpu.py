"""Mixed types under autocast: the library products of an operator take autocast's type, its kernels one type for all operands.
Bounds: a chain of at most eight roundings to bf16 (2^-9 each, in the 2-norm)."""

import pytest
import torch
from torch.nn import functional as F

import oops_b200 as oops

pytestmark = pytest.mark.gpu


def close(got, want, bound=8 * 2.0**-9):
    for a, b in zip(got, want):
        assert a.shape == b.shape
        assert float((a.double() - b.double()).norm()) <= bound * float(b.double().norm())


def gate_operands(device, dtype):
    gen = torch.Generator().manual_seed(3)
    shapes = ((2, 2, 40, 16), (2, 40, 24), (32, 24), (24, 32))
    return [(0.5 * torch.randn(*s, generator=gen)).to(device, dtype).requires_grad_(True) for s in shapes]


def composed(attention, single, gate_weight, output_weight):
    values = attention.transpose(-2, -3).flatten(-2)
    return F.linear(torch.sigmoid(F.linear(single, gate_weight)) * values, output_weight)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("region", [torch.bfloat16, torch.float16])
def test_gate_output_forward_under_autocast(cuda, dtype, region):
    leaves = gate_operands(cuda, dtype)
    with torch.autocast("cuda", dtype=region):
        out = oops.gate_attention_output(*leaves)
    assert out.dtype is region
    exact = [t.detach().double().requires_grad_(True) for t in leaves]
    want = composed(*exact)
    close([out], [want])
    close(torch.autograd.grad(out, leaves, torch.ones_like(out)), torch.autograd.grad(want, exact, torch.ones_like(want)))


def test_gate_output_reverse_under_autocast(cuda):
    leaves = gate_operands(cuda, torch.float32)
    want = torch.autograd.grad(oops.gate_attention_output(*leaves).sum(), leaves)
    total = oops.gate_attention_output(*leaves).sum()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        got = torch.autograd.grad(total, leaves)
    close(got, want, 0.0)


def test_pair_update_reverse_under_autocast(cuda):
    gen = torch.Generator().manual_seed(4)
    names = ("input_norm_weight", "input_norm_bias", "output_norm_weight", "output_norm_bias", "left_gate_weight", "left_value_weight",
             "right_gate_weight", "right_value_weight", "output_gate_weight", "output_weight")
    weights = {n: (0.3 * torch.randn(*((16,) if "norm" in n else (16, 16)), generator=gen)).to(cuda).requires_grad_(True) for n in names}
    pair = torch.randn(1, 12, 12, 16, generator=gen).to(cuda).requires_grad_(True)
    leaves = [pair, *weights.values()]
    want = torch.autograd.grad(oops.triangle_multiplication(pair, **weights).sum(), leaves)
    total = oops.triangle_multiplication(pair, **weights).sum()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        got = torch.autograd.grad(total, leaves)
    close(got, want, 0.0)
