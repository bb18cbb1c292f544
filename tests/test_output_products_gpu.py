"""The output step of token attention on this library's own products, at the edges of their 128 x 64 x 64 tiles: fewer rows than a tile, ragged
rows, channels and products, heads of 8 and 24 channels, head- and token-major values, subsets of the gradients; and beside it the sizes
and layouts that stay with the library's products.  Against f64: the gate, the gated values and the results are rounded to 16 bits
(half a unit each: 2^-9 bf16, 2^-12 f16 of their magnitude), their sums in f32; the norm of the error is that of some four
independent roundings, of which each is at most half a unit."""

import pytest
import torch

from oops_b200 import gate_attention_output
from oops_b200.runtime import cabi

pytestmark = pytest.mark.gpu
ROUNDING = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}


def operands(dtype, samples, heads, tokens, dim, channels, out, device):
    gen = torch.Generator().manual_seed(tokens * dim + channels)

    def normal(*shape, scale=1.0):
        return (scale * torch.randn(shape, generator=gen)).to(dtype).to(device)

    inner = heads * dim
    return [normal(samples, heads, tokens, dim), normal(samples, tokens, channels), normal(inner, channels, scale=channels**-0.5),
            normal(out, inner, scale=inner**-0.5)], normal(samples, tokens, out)


@pytest.mark.parametrize("dtype,samples,heads,tokens,dim,channels,out,layout",
                         [(torch.bfloat16, 1, 1, 1, 8, 8, 8, "head"), (torch.bfloat16, 2, 3, 65, 24, 72, 40, "head"),
                          (torch.float16, 3, 2, 43, 64, 64, 136, "token"), (torch.bfloat16, 1, 2, 257, 16, 200, 64, "head"),
                          (torch.bfloat16, 2, 4, 50, 16, 47, 31, "head"),  # channels that are no words: the library's products
                          (torch.float16, 1, 16, 2100, 64, 384, 384, "head")])  # as many rows as the own products take, nearly
def test_forward_and_reverse(cuda, dtype, samples, heads, tokens, dim, channels, out, layout):
    tensors, up = operands(dtype, samples, heads, tokens, dim, channels, out, cuda)
    if layout == "token":
        tensors[0] = tensors[0].transpose(1, 2).contiguous().transpose(1, 2)
    leaves = [t.detach().requires_grad_(True) for t in tensors]
    got = gate_attention_output(*leaves)
    grads = torch.autograd.grad(got, leaves, up, retain_graph=True)
    exact = [t.double().requires_grad_(True) for t in tensors]
    gated = torch.sigmoid(exact[1] @ exact[2].t()) * exact[0].transpose(1, 2).flatten(-2)
    want = gated @ exact[3].t()
    for have, ref in zip((got, *grads), (want, *torch.autograd.grad(want, exact, up.double()))):
        have, ref = have.detach().double(), ref.detach()
        assert float((have - ref).norm()) <= 2 * ROUNDING[dtype] * float(ref.norm())
    for leaf, all_at_once in zip(leaves, grads):  # each alone takes other lists of products
        alone, = torch.autograd.grad(got, [leaf], up, retain_graph=True)
        assert torch.equal(alone, all_at_once)
    with torch.no_grad():
        assert torch.equal(gate_attention_output(*leaves), got.detach())
    assert cabi.library().oops_ta_device_status(0) == 0


def test_repeated_calls_agree_bit_for_bit(cuda):
    tensors, up = operands(torch.bfloat16, 4, 16, 512, 64, 384, 384, cuda)
    leaves = [t.requires_grad_(True) for t in tensors]

    def run():
        got = gate_attention_output(*leaves)
        return [got.detach(), *torch.autograd.grad(got, leaves, up)]

    first = run()
    for _ in range(40):
        assert all(torch.equal(a, b) for a, b in zip(first, run()))


@pytest.mark.parametrize("dtype,rows,heads,dim,channels,out", [
    (torch.bfloat16, 512, 1, 8, 8, 8),       # eight steps of the weights' gradients: one part; one tile
    (torch.bfloat16, 513, 3, 24, 72, 40),    # nine: two parts, the last step of one row
    (torch.float16, 1025, 2, 64, 136, 200),  # 17: four parts; tiles that leave places of a cluster empty
    (torch.bfloat16, 2049, 4, 24, 520, 72),  # 33: eight parts; nine steps forward
    (torch.float16, 40, 32, 64, 1000, 712),  # 16 and 32 steps forward: two and four parts
    (torch.bfloat16, 7, 4, 8, 4104, 2056),   # 65 steps forward and 33 in the reverse
    (torch.bfloat16, 16000, 2, 8, 128, 64),  # 250 steps: parts of 31 and 32
    (torch.float16, 768, 16, 64, 384, 384),  # 36 tiles in four parts: more CTAs than clusters of them find SMs for
    (torch.bfloat16, 2400, 16, 64, 384, 384),  # more work, rows or weights than the own products take: the library's
    (torch.bfloat16, 32776, 1, 8, 8, 8),
    (torch.bfloat16, 16, 32, 64, 768, 64),
])
def test_sums_in_parts(cuda, dtype, rows, heads, dim, channels, out):
    """Sums over more steps than a part takes are made by the CTAs of a cluster and added in their order."""
    tensors, up = operands(dtype, 1, heads, rows, dim, channels, out, cuda)
    leaves = [t.detach().requires_grad_(True) for t in tensors]
    got = gate_attention_output(*leaves)
    grads = torch.autograd.grad(got, leaves, up, retain_graph=True)
    exact = [t.double().requires_grad_(True) for t in tensors]
    want = (torch.sigmoid(exact[1] @ exact[2].t()) * exact[0].transpose(1, 2).flatten(-2)) @ exact[3].t()
    for have, ref in zip((got, *grads), (want, *torch.autograd.grad(want, exact, up.double()))):
        have, ref = have.detach().double(), ref.detach()
        assert float((have - ref).norm()) <= 2 * ROUNDING[dtype] * float(ref.norm())
    for leaf, all_at_once in zip(leaves, grads):
        for _ in range(3):
            alone, = torch.autograd.grad(got, [leaf], up, retain_graph=True)
            assert torch.equal(alone, all_at_once)
    assert cabi.library().oops_ta_device_status(0) == 0
