"""Forward calls without a mask that give a CTA several items: one and several key steps, ragged ends, an odd number of rows
(the last row is its own partner), with and without the gate.  16-bit bounds as in the parity tests: 2e-2 of the largest value
(at least 1); the statistics are checked through the gradients of the rows on either side of an item's end."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention, triangle_attention_gated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,batch,rows,n,heads,bias_kind",
                         [(torch.bfloat16, 1, 155, 64, 4, "shared"), (torch.float16, 2, 151, 40, 4, "none"),
                          (torch.bfloat16, 1, 149, 130, 4, "shared"), (torch.bfloat16, 1, 303, 257, 2, "shared"),
                          (torch.float16, 1, 640, 128, 1, "shared")])
def test_several_items_per_cta(cuda, dtype, batch, rows, n, heads, bias_kind):
    gen = torch.Generator().manual_seed(rows)
    q, k, v, gate, up = (torch.randn(batch, rows, n, heads, 32, generator=gen).to(dtype) for _ in range(5))
    bias = (4 * torch.randn(batch, 1, heads, n, n, generator=gen)).to(dtype) if bias_kind == "shared" else None
    want = oracle.forward_backward(q, k, v, None, bias, up)
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v)]
    on = None if bias is None else bias.to(cuda)
    out = triangle_attention(*leaves, None, on)
    grads = torch.autograd.grad(out, leaves, up.to(cuda))
    for name, got, ref in zip(("out", "dq", "dk", "dv"), (out, *grads), want):
        error = float((got.detach().float().cpu() - ref).abs().max())
        assert error <= 2e-2 * max(1.0, float(ref.abs().max())), (name, error)
    with torch.no_grad():
        gated = triangle_attention_gated(*(t.detach() for t in leaves), gate.to(cuda), None, on)
    expect = torch.sigmoid(gate.float()) * want[0]
    assert float((gated.float().cpu() - expect).abs().max()) <= 2e-2 * max(1.0, float(expect.abs().max()))
