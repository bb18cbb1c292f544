"""The f32 kernels that keep their scores on chip, at the sizes where their 64 x 64 tiles and channel groups end, with each
kind of bias and with masks that drop whole tiles and whole rows; against the oracle in f64.  A result is a sum of at most
cols + dim products with f32 rounding (2^-24) in every one of them and in its weights: (cols + dim) * 2^-22 of the largest
value bounds it with a factor of four to spare."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention
from oops_b200.runtime import cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols,dim,bias_kind,mask_kind,swapped",
                         [(1, 32, "none", "none", False), (63, 1, "shared", "random", False), (64, 32, "shared", "ones", False),
                          (65, 30, "full", "tokens", False), (130, 16, "shared", "tokens", True), (200, 64, "shared", "random", True),
                          (97, 33, "none", "random", False)])
def test_tile_edges(cuda, cols, dim, bias_kind, mask_kind, swapped):
    gen = torch.Generator().manual_seed(cols)
    rows, heads = (cols, 4) if swapped else (40, 2)  # at least 74 (row, head) pairs: the one-pass reverse kernel
    shape = (1, rows, cols, heads, dim)
    q, k, v, up = (torch.randn(shape, generator=gen) for _ in range(4))
    bias = None if bias_kind == "none" else torch.randn(1, 1 if bias_kind == "shared" else rows, heads, cols, cols, generator=gen)
    mask = {"none": None, "ones": torch.ones(1, rows, cols, dtype=torch.bool),
            "random": torch.rand(1, rows, cols, generator=gen) > 0.3,
            "tokens": ((torch.arange(cols) < max(1, cols // 2 - 3)) & (torch.arange(rows)[:, None] > 2))[None]}[mask_kind]
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v)] + ([] if bias is None else [bias.to(cuda).requires_grad_(True)])
    views = [t.transpose(1, 2).contiguous().transpose(1, 2) if swapped else t for t in leaves[:3]]  # column-major storage
    out = triangle_attention(*views, None if mask is None else mask.to(cuda), None if bias is None else leaves[3])
    grads = torch.autograd.grad(out, leaves, up.to(cuda))
    ref = [t.double().requires_grad_(True) for t in (q, k, v)] + ([] if bias is None else [bias.double().requires_grad_(True)])
    want = oracle.reference_dense(ref[0], ref[1], ref[2], mask, None if bias is None else ref[3], compute_dtype=torch.float64)
    want_grads = torch.autograd.grad(want, ref, up.double())
    for name, got, exact in zip(("out", "dq", "dk", "dv", "dbias"), (out, *grads), (want, *want_grads)):
        terms = cols + dim + (rows if name == "dbias" else 0)
        bound = terms * 2.0**-22 * max(1.0, float(exact.detach().abs().max()))
        assert float((got.detach().double().cpu() - exact.detach()).abs().max()) <= bound, name
    if mask is not None:
        empty = ~mask.any(-1)
        assert torch.count_nonzero(out.detach().cpu()[empty]) == 0


def test_bias_gradient_over_several_launches(cuda):
    """832 columns of 4 heads: 24 rows of dS fit the scratch of a launch, so 30 rows take two, and the second adds."""
    gen = torch.Generator().manual_seed(1)
    rows, cols, heads, dim = 30, 832, 4, 8
    q, k, v, up = (torch.randn(1, rows, cols, heads, dim, generator=gen) for _ in range(4))
    bias = torch.randn(1, 1, heads, cols, cols, generator=gen)
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v, bias)]
    out = triangle_attention(*leaves[:3], None, leaves[3])
    before = cabi.launch_count()
    grads = torch.autograd.grad(out, leaves, up.to(cuda))
    assert cabi.launch_count() - before == 4  # a reverse pass and a sum per launch
    ref = [t.to(cuda, torch.float64).requires_grad_(True) for t in (q, k, v, bias)]
    want = oracle.reference_dense(*ref[:3], None, ref[3], compute_dtype=torch.float64)
    for name, got, exact in zip(("dq", "dk", "dv", "dbias"), grads, torch.autograd.grad(want, ref, up.to(cuda, torch.float64))):
        bound = (cols + dim + rows) * 2.0**-22 * max(1.0, float(exact.abs().max()))
        assert float((got.double() - exact).abs().max()) <= bound, name
