"""The tcgen05 forward kernel takes its softmax reference from a row's first step and raises it only when a later step's
sum asks for it: logits that climb by far more than the f16 and bf16 ranges, fall, jump inside a step, or stay below
any reference for whole steps; masks whose first kept key comes late, whose kept keys are scattered over few steps, or that
drop rows; odd row counts (a CTA with one tile) and one row (query tiles paired instead of rows).  Against the oracle in
f64: probabilities and the result are rounded to 16 bits, 2^-9 (bf16) or 2^-12 (f16) of values that reach max|v|, twice."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention

pytestmark = pytest.mark.gpu
ROUNDING = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}


def _bias(kind, rows, heads, n, gen):
    key = torch.arange(n, dtype=torch.float32)
    base = {"climbing": key * 0.9, "falling": -key * 0.9, "spike": 150.0 * (key == n - 3), "steps": 40.0 * (key // 64),
            "flat": torch.zeros(n), "low": torch.where(key < 64, torch.full((n,), -200.0), torch.zeros(n))}[kind]
    return base + 0.25 * torch.randn(1, rows, heads, n, n, generator=gen)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind,rows,n,mask_kind,full",
                         [("climbing", 3, 200, "none", False), ("falling", 2, 130, "none", False), ("spike", 5, 328, "late", False),
                          ("steps", 1, 264, "none", False), ("flat", 4, 256, "scattered", False), ("low", 3, 192, "rows", False),
                          ("climbing", 3, 392, "late", True), ("spike", 1, 64, "none", False), ("flat", 7, 72, "rows", True)])
def test_references(cuda, dtype, kind, rows, n, mask_kind, full):
    gen = torch.Generator().manual_seed(n)
    heads = 2
    q, k, v = ((0.5 * torch.randn(1, rows, n, heads, 32, generator=gen)).to(dtype) for _ in range(3))
    bias = _bias(kind, rows if full else 1, heads, n, gen).to(dtype)
    mask = None
    if mask_kind == "late":
        mask = (torch.arange(n) >= n - 70).expand(1, rows, n).clone()
        mask[:, 0] = True
    elif mask_kind == "scattered":
        mask = ((torch.arange(n) % 97) == 5).expand(1, rows, n).clone()
        mask[:, 1, :] = torch.arange(n) == 200
    elif mask_kind == "rows":
        mask = torch.rand(1, rows, n, generator=gen) > 0.5
        mask[:, 1] = False
    if mask is not None:
        k, v = k.masked_fill(~mask[..., None, None], float("inf")), v.masked_fill(~mask[..., None, None], float("nan"))
    with torch.no_grad():
        out = triangle_attention(q.to(cuda), k.to(cuda), v.to(cuda), None if mask is None else mask.to(cuda), bias.to(cuda))
    want = oracle.reference_dense(q.double(), torch.nan_to_num(k.double(), posinf=0.0), torch.nan_to_num(v.double(), nan=0.0), mask,
                                  bias.double(), compute_dtype=torch.float64)
    error = float((out.double().cpu() - want).abs().max())
    assert error <= 2 * ROUNDING[dtype] * float(torch.nan_to_num(v.double(), nan=0.0).abs().max()), error
    if mask is not None:
        assert torch.count_nonzero(out.cpu()[~mask.any(-1)]) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,n,column", [(60, 64, 40), (60, 136, 63), (1, 512, 17), (40, 100, 30)])
def test_the_largest_probability_of_the_first_step_is_exact(cuda, dtype, rows, n, column):
    """One key of the first step carries 0.6 to 0.95 of every row.  Its probability is the reference, 1 before the division by
    the sum, so the result is off by its own rounding and the rounding of the light keys: less than 1.15 of the result's
    rounding in the 2-norm, where a rounded largest probability makes it 1.4."""
    gen = torch.Generator().manual_seed(n)
    heads = 2
    q, k, v = ((0.5 * torch.randn(1, rows, n, heads, 32, generator=gen)).to(dtype) for _ in range(3))
    bias = torch.randn(1, 1, heads, n, n, generator=gen)
    bias[..., column] += 2.0 + torch.log(torch.tensor(float(n)))
    bias = bias.to(dtype)
    with torch.no_grad():
        out = triangle_attention(q.to(cuda), k.to(cuda), v.to(cuda), None, bias.to(cuda)).double().cpu()
    want = oracle.reference_dense(q.double(), k.double(), v.double(), None, bias.double(), compute_dtype=torch.float64)
    rounding = float((want.to(dtype).double() - want).norm())
    assert float((out - want).norm()) <= 1.15 * rounding
