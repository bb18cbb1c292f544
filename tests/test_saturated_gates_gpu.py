"""The gate of the output step and its slope one value at a time, where it is saturated: operands are laid out so that every product has one
term that is not zero (a row of ones and zeros in, the identity behind), so that results are gate values rounded once.

Bound: half a unit of the type (2^-11 f16, 2^-8 bf16, relative), and 2^-15 for f32 arithmetic: exp(-|g|) is off by the rounding of its exponent,
|g| log2(e) 2^-24 ln 2 < 1.1e-6 for |g| <= 16, and by 2 units of 2^-23; the rest are a few roundings."""

import pytest
import torch

from oops_b200 import gate_attention_output

pytestmark = pytest.mark.gpu
HALF_UNIT = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_saturated_gates(cuda, dtype):
    heads, dim = 16, 64
    inner = heads * dim
    gates = torch.linspace(-16, 16, inner, device=cuda).to(dtype)
    gate_weight = torch.zeros(inner, 8, device=cuda, dtype=dtype)
    gate_weight[:, 0] = gates
    gate_weight.requires_grad_(True)
    single = torch.zeros(1, 1, 8, device=cuda, dtype=dtype)
    single[..., 0] = 1
    attention = torch.full((1, heads, 1, dim), 64.0, device=cuda, dtype=dtype).requires_grad_(True)  # (keeps f16 results in its normal range)
    upstream = torch.full((1, 1, inner), 32.0, device=cuda, dtype=dtype)
    out = gate_attention_output(attention, single, gate_weight, torch.eye(inner, device=cuda, dtype=dtype))
    dattention, dgate = torch.autograd.grad(out, [attention, gate_weight], upstream)
    g = gates.double()
    s = torch.sigmoid(g)
    slope = s * torch.sigmoid(-g)
    for name, got, want in (("gated", out.flatten(), 64 * s), ("values", dattention.flatten(), 32 * s), ("gate", dgate[:, 0], 2048 * slope)):
        normal = want > torch.finfo(dtype).tiny
        assert int(normal.sum()) > inner * 3 // 4
        error = ((got.detach().double() - want).abs() / want)[normal]
        assert float(error.max()) <= HALF_UNIT[dtype] + 2.0**-15, name
    assert bool((dgate[:, 1:] == 0).all())


def test_gates_beyond_every_exponent(cuda):
    """exp(-|g|) underflows, or the gate is not a number: one and zero, and a NaN that stays one."""
    heads, dim = 1, 8
    gates = torch.tensor([200.0, -200.0, float("inf"), -float("inf"), float("nan"), 0.0, -87.5, 87.5], device=cuda).bfloat16()
    attention = torch.ones(1, heads, 1, dim, device=cuda).bfloat16().requires_grad_(True)
    single = torch.ones(1, 1, 8, device=cuda).bfloat16()
    weight = torch.zeros(8, 8, device=cuda).bfloat16()
    weight[:, 0] = gates
    single[..., 1:] = 0
    weight.requires_grad_(True)
    out = gate_attention_output(attention, single, weight, torch.eye(8, device=cuda).bfloat16())
    seen = [gate_attention_output(attention, single, weight[i : i + 1].repeat(8, 1), torch.eye(8, device=cuda).bfloat16()).flatten()[0] for i in range(8)]
    assert torch.isnan(out).all()  # (the identity's zeros meet the NaN)
    want = torch.sigmoid(gates.double())
    for got, ref in zip(seen, want):
        if torch.isnan(ref):
            assert torch.isnan(got)
        else:
            assert abs(float(got) - float(ref)) <= 2.0**-8 * float(ref) + 2.0**-133  # (half of the smallest bf16 is 2^-134)
