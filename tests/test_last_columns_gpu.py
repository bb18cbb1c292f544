"""The last 16 columns of a step, which the tcgen05 forward kernel looks at before it has their probabilities: one large logit there and nowhere else, below and
above what sends a step back for a new reference (2^10 of the reference's probability; 2^6 once was the limit) and far beyond the range of 16 bits and of f32,
in steps of every walk (one row, pairs of rows, several items of a CTA, steps without tests behind a mask, steps with tests).
Against the oracle in f64: probabilities and the result are rounded to 16 bits, 2^-9 (bf16) or 2^-12 (f16) of values that reach max|v|, twice."""

import math

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention

pytestmark = pytest.mark.gpu
ROUNDING = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("walk", ["row", "pairs", "items", "masked", "tests"])
@pytest.mark.parametrize("height", [5.5, 6.5, 9.5, 10.5, 18.0, 200.0])
def test_one_large_logit(cuda, dtype, walk, height):
    gen = torch.Generator().manual_seed(int(height * 10))
    rows, n, heads = {"row": 1, "pairs": 3, "items": 330, "masked": 3, "tests": 3}[walk], 320 if walk != "items" else 192, 1
    q, k, v = ((0.5 * torch.randn(1, rows, n, heads, 32, generator=gen)).to(dtype) for _ in range(3))
    bias = 0.25 * torch.randn(1, 1, heads, n, n, generator=gen)
    for query in range(n):  # every one of the 16 columns, of the second and the last but one step
        bias[..., query, (64 if query % 2 else n - 128) + 48 + query // 2 % 16] += height * math.log(2.0)
    bias = bias.to(dtype)
    mask = None
    if walk == "masked":  # the last step is left out, and a key of the first
        mask = (torch.arange(n) < n - 64).expand(1, rows, n).clone()
        mask[..., 3] = False
    elif walk == "tests":
        mask = torch.ones(1, rows, n, dtype=torch.bool)
        mask[..., 5::64] = False
    with torch.no_grad():
        out = triangle_attention(q.to(cuda), k.to(cuda), v.to(cuda), None if mask is None else mask.to(cuda), bias.to(cuda)).double().cpu()
    want = oracle.reference_dense(q.double(), k.double(), v.double(), mask, bias.double(), compute_dtype=torch.float64)
    assert float((out - want).abs().max()) <= 2 * ROUNDING[dtype] * float(v.double().abs().max())
