"""The row dots and the look at the mask that precede the reverse kernels: heads that leave lanes of a group of four idle, rows that are no
multiple of the mask's batches of 512 keys, kept prefixes that end on either side of one, pair axes exchanged in memory.  16-bit bounds
as in the parity tests: 2e-2 of the largest value (at least 1)."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,rows,cols,heads,kept,swapped", [(torch.bfloat16, 3, 40, 1, None, False), (torch.float16, 9, 130, 3, 129, False),
                                                                (torch.bfloat16, 2, 600, 5, 511, False), (torch.bfloat16, 2, 600, 6, 512, True),
                                                                (torch.float16, 2, 520, 2, 513, False), (torch.bfloat16, 17, 72, 4, 1, True)])
def test_gradients(cuda, dtype, rows, cols, heads, kept, swapped):
    gen = torch.Generator().manual_seed(cols + heads)
    q, k, v, up = (torch.randn(1, rows, cols, heads, 32, generator=gen).to(dtype) for _ in range(4))
    bias = torch.randn(1, 1, heads, cols, cols, generator=gen).to(dtype)
    mask = None if kept is None else (torch.arange(cols) < kept).expand(1, rows, cols).contiguous()
    if kept is not None and rows > 8:
        mask[:, ::2, 0] = False  # (other rows of a block of eight keep a prefix)
    want = oracle.forward_backward(q, k, v, mask, bias, up)

    def laid_out(t):
        t = t.to(cuda)
        return t.transpose(1, 2).contiguous().transpose(1, 2) if swapped else t

    leaves = [laid_out(t).detach().requires_grad_(True) for t in (q, k, v)] + [bias.to(cuda).requires_grad_(True)]
    out = triangle_attention(*leaves[:3], None if mask is None else mask.to(cuda), leaves[3])
    grads = torch.autograd.grad(out, leaves, laid_out(up))
    for name, got, ref in zip(("out", "dq", "dk", "dv", "dbias"), (out, *grads), want):
        error = float((got.detach().float().cpu() - ref).abs().max())
        assert error <= 2e-2 * max(1.0, float(ref.abs().max())), (name, error)


@pytest.mark.parametrize("dtype,rows,cols,heads,kept,swapped", [(torch.bfloat16, 40, 130, 1, 129, False), (torch.float16, 10, 520, 1, None, True),
                                                                (torch.bfloat16, 20, 268, 1, None, False), (torch.float16, 20, 284, 1, 280, False),
                                                                (torch.bfloat16, 12, 196, 2, None, False)])
def test_one_head(cuda, dtype, rows, cols, heads, kept, swapped):
    """One head, whose dots have an instance of their own; bias gradients on either side of where their parts are added four keys a thread."""
    test_gradients(cuda, dtype, rows, cols, heads, kept, swapped)
