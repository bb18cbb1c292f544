"""The tcgen05 kernels for bf16 operands with head sizes up to 64, at the sizes where their 128-row tiles, 64-column steps and
16-channel groups end: one and several steps, ragged ones, head sizes that pad, several parts of the bias gradient, a bias per
row, subsets of the gradients; against the oracle in f64.  Products carry 16 mantissa bits, so the forward result is off by its
own rounding (half a unit: 2^-9 of the largest value; twice that is allowed); the gradients see the rounded output through
delta = sum(out * dout), whose error is that rounding times |dout| summed over the head (sqrt(64) at most): eight times the forward
bound."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import pair_bias_attention, triangle_attention
from oops_b200.runtime import cabi

pytestmark = pytest.mark.gpu
ROUNDING = 2.0**-8


def close(name, got, exact):
    got, exact = got.detach().double().cpu(), exact.detach()
    bound = ROUNDING * (1 if name == "out" else 8) * max(1.0, float(exact.abs().max()))
    error = float((got - exact).abs().max())
    assert error <= bound, (name, error, bound)


@pytest.mark.parametrize("rows,cols,heads,dim,bias_kind",
                         [(3, 1, 2, 64, "none"), (2, 8, 3, 64, "shared"), (2, 65, 2, 64, "shared"), (3, 63, 2, 48, "none"),
                          (2, 128, 2, 40, "shared"), (1, 129, 1, 64, "shared"), (20, 130, 2, 8, "shared"), (2, 192, 2, 16, "row"),
                          (3, 257, 1, 24, "shared"), (2, 320, 2, 56, "row"), (1, 449, 2, 64, "none")])
def test_tile_edges(cuda, rows, cols, heads, dim, bias_kind):
    gen = torch.Generator().manual_seed(cols)
    shape = (1, rows, cols, heads, dim)
    q, k, v, up = (torch.randn(shape, generator=gen).bfloat16() for _ in range(4))
    groups = {"none": 0, "shared": 1, "row": rows}[bias_kind]
    bias = (3 * torch.randn(1, groups, heads, cols, cols, generator=gen)).bfloat16() if groups else None
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v)]
    on = bias.to(cuda).requires_grad_(groups == 1) if groups else None  # (the gradient of a bias per row is made elsewhere)
    out = triangle_attention(*leaves, None, on)
    wanted = leaves + ([on] if groups == 1 else [])
    grads = torch.autograd.grad(out, wanted, up.to(cuda), retain_graph=True)
    ref = [t.double().requires_grad_(True) for t in (q, k, v)] + ([bias.double().requires_grad_(True)] if groups else [])
    want = oracle.reference_dense(ref[0], ref[1], ref[2], None, ref[3] if groups else None, compute_dtype=torch.float64)
    want_grads = torch.autograd.grad(want, ref[:len(wanted)], up.double())
    for name, got, exact in zip(("out", "dq", "dk", "dv", "dbias"), (out, *grads), (want, *want_grads)):
        close(name, got, exact)
    for leaf, all_at_once in zip(wanted, grads):  # each alone: the other kinds of CTA are not launched
        alone, = torch.autograd.grad(out, [leaf], up.to(cuda), retain_graph=True)
        assert torch.equal(alone, all_at_once)
    assert cabi.library().oops_ta_device_status(0) == 0


def test_head_major_operands(cuda):
    """Token attention's own layout, and a gradient whose rows are no 16-byte words."""
    gen = torch.Generator().manual_seed(7)
    q, k, v, up = (torch.randn(2, 4, 201, 48, generator=gen).bfloat16() for _ in range(4))
    bias = torch.randn(1, 4, 201, 201, generator=gen).bfloat16()
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v, bias)]
    out = pair_bias_attention(*leaves[:3], pair_bias=leaves[3])
    grads = torch.autograd.grad(out, leaves, up.to(cuda))
    ref = [t.double().requires_grad_(True) for t in (q, k, v, bias)]
    want = torch.softmax(ref[0] @ ref[1].transpose(-1, -2) * 48**-0.5 + ref[3], -1) @ ref[2]
    for name, got, exact in zip(("out", "dq", "dk", "dv", "dbias"), (out, *grads), (want, *torch.autograd.grad(want, ref, up.double()))):
        close(name, got, exact)


@pytest.mark.parametrize("cols", [192, 512])
def test_repeated_calls_agree_bit_for_bit(cuda, cols):
    """Many CTAs beside each other, three and eight steps: a read ahead of the last product's end shows up here as rows that differ."""
    gen = torch.Generator().manual_seed(cols)
    leaves = [torch.randn(4, 16, cols, 64, generator=gen).bfloat16().to(cuda).requires_grad_(True) for _ in range(3)]
    bias = torch.randn(1, 16, cols, cols, generator=gen).bfloat16().to(cuda).requires_grad_(True)
    up = torch.randn(4, 16, cols, 64, generator=gen).bfloat16().to(cuda)

    def run():
        out = pair_bias_attention(*leaves, pair_bias=bias)
        return [out.detach(), *torch.autograd.grad(out, [*leaves, bias], up)]

    first = run()
    for _ in range(40):
        assert all(torch.equal(a, b) for a, b in zip(first, run()))
