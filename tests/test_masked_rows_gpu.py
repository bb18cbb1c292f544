"""Masks that drop whole key tiles and whole rows: the tcgen05 kernels pass them over.  Every gradient must be what the oracle
says, exact zeros where nothing is kept, whatever the dropped operands hold; one and several groups of query tiles per row,
more and fewer (row, head) items than SMs, rows whose live tiles have gaps,
and masks that keep everything or all but one key (they choose the walk without tests).  16-bit bounds as in the parity tests: 2e-2 of
the largest value (at least 1)."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,rows,n,heads,mask_kind,bias_kind",
                         [(torch.bfloat16, 90, 300, 4, "tokens", "shared"), (torch.float16, 7, 136, 2, "gaps", "none"),
                          (torch.bfloat16, 5, 1000, 2, "tokens", "shared"), (torch.bfloat16, 40, 264, 4, "gaps", "shared"),
                          (torch.bfloat16, 9, 392, 2, "all dropped", "shared"), (torch.float16, 160, 72, 2, "tokens", "shared"),
                          (torch.bfloat16, 90, 256, 2, "nothing dropped", "shared"), (torch.bfloat16, 90, 256, 2, "one key", "shared"),
                          (torch.float16, 3, 1024, 2, "nothing dropped", "shared"), (torch.float16, 3, 1024, 2, "one key", "none")])
def test_gradients(cuda, dtype, rows, n, heads, mask_kind, bias_kind):
    gen = torch.Generator().manual_seed(n)
    q, k, v = ((0.5 * torch.randn(1, rows, n, heads, 32, generator=gen)).to(dtype) for _ in range(3))
    up = torch.randn(1, rows, n, heads, 32, generator=gen).to(dtype)
    bias = torch.randn(1, 1, heads, n, n, generator=gen).to(dtype) if bias_kind == "shared" else None
    if mask_kind == "tokens":
        mask = ((torch.arange(n) < n // 2 - 5) & (torch.arange(rows)[:, None] < rows - rows // 3))[None]
    elif mask_kind == "gaps":  # a different pattern of 128-key tiles in every row
        tile = torch.arange(n) // 128
        mask = ((torch.arange(rows)[:, None] >> tile) & 1).bool()[None] & (torch.rand(1, rows, n, generator=gen) > 0.2)
    else:
        mask = torch.full((1, rows, n), mask_kind != "all dropped")
        mask[0, -1, -1] = mask_kind == "nothing dropped"
    k, v = k.masked_fill(~mask[..., None, None], float("inf")), v.masked_fill(~mask[..., None, None], float("nan"))
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v)] + ([] if bias is None else [bias.to(cuda).requires_grad_(True)])
    out = triangle_attention(*leaves[:3], mask.to(cuda), leaves[3] if bias is not None else None)
    grads = torch.autograd.grad(out, leaves, up.to(cuda))
    want = oracle.forward_backward(q, torch.nan_to_num(k, posinf=0.0), torch.nan_to_num(v, nan=0.0), mask, bias, up)
    for name, got, ref in zip(("out", "dq", "dk", "dv", "dbias"), (out, *grads), want):
        error = float((got.detach().float().cpu() - ref).abs().max())
        assert error <= 2e-2 * max(1.0, float(ref.abs().max())), (name, error)
    empty = ~mask.any(-1)
    for got in (out.detach(), grads[0]):
        assert torch.count_nonzero(got.cpu()[empty]) == 0
    for got in grads[1:3]:
        assert torch.count_nonzero(got.cpu()[~mask]) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,n,full", [(6, 256, False), (5, 328, False), (4, 200, True), (1, 392, False)])
def test_steps_that_only_one_row_of_a_pair_keeps(cuda, dtype, rows, n, full):
    """Neighbouring rows keep alternate blocks of 64 keys, and one row keeps none at all: each walks steps that only its
    partner keeps.  Bound: probabilities and result rounded to 16 bits, of values that reach max|v|, twice."""
    from oracle import triangle_oracle as oracle

    gen = torch.Generator().manual_seed(n)
    heads = 2
    q, k, v = ((0.5 * torch.randn(1, rows, n, heads, 32, generator=gen)).to(dtype) for _ in range(3))
    bias = torch.randn(1, rows if full else 1, heads, n, n, generator=gen).to(dtype)
    mask = ((torch.arange(n) // 64 + torch.arange(rows)[:, None]) % 2 == 0)[None].clone()
    mask[:, 3:4] = False
    k, v = k.masked_fill(~mask[..., None, None], float("inf")), v.masked_fill(~mask[..., None, None], float("nan"))
    with torch.no_grad():
        out = triangle_attention(q.to(cuda), k.to(cuda), v.to(cuda), mask.to(cuda), bias.to(cuda)).double().cpu()
    finite = torch.nan_to_num(v.double(), nan=0.0)
    want = oracle.reference_dense(q.double(), torch.nan_to_num(k.double(), posinf=0.0), finite, mask, bias.double(), compute_dtype=torch.float64)
    bound = 2 * (2.0**-8 if dtype is torch.bfloat16 else 2.0**-11) * float(finite.abs().max())
    assert float((out - want).abs().max()) <= bound
    assert torch.count_nonzero(out[~mask.any(-1)]) == 0
