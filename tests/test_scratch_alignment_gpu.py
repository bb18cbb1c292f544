"""The bias gradient alone, from scratch memory that starts off a 16-byte boundary: bit for bit what aligned scratch gives (the sums of its parts
have an order, whichever width they are read in)."""

import pytest
import torch

from oops_b200.attention.triangle import function as fn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [32, 64])
@pytest.mark.parametrize("cols", [136, 256])
@pytest.mark.parametrize("offset", [4, 8])
def test_bias_gradient(cuda, dim, cols, offset):
    gen = torch.Generator().manual_seed(cols)
    rows, heads, want = 20, 2, (False, False, False, True)
    q, k, v, up = (torch.randn(1, rows, cols, heads, dim, generator=gen).to(cuda, torch.bfloat16) for _ in range(4))
    bias = torch.randn(1, 1, heads, cols, cols, generator=gen).to(cuda, torch.bfloat16)
    geometry, scale = fn.DenseGeometry(), dim**-0.5
    out, lse = fn.run_forward(geometry, q, k, v, None, bias, scale, 0, True)
    size = fn.backward_scratch_bytes(q, k, v, None, bias, scale, 0, want)
    memory = torch.empty(size + 16, dtype=torch.uint8, device=cuda)

    def call(scratch):
        return [g for g in fn.run_backward(geometry, up, q, k, v, None, bias, out, lse, scale, 0, want, scratch=scratch) if g is not None]

    assert memory.data_ptr() % 16 == 0 and size > 8 * rows * heads * cols  # (several parts)
    for got, expected in zip(call(memory[offset : offset + size]), call(memory[:size])):
        assert torch.equal(got, expected)
