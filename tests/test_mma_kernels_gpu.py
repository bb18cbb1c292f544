"""The 16-bit kernels for head sizes and layouts the tcgen05 kernels do not take, at the sizes where their 64 x 64 tiles and
16-channel groups end: head sizes that are no multiple of 8, unaligned rows, f32 biases, masks that drop tiles and rows,
several parts of the bias gradient; against the oracle in f64.  Products are exact or carry 16 mantissa bits, so the forward
result is off by its own rounding (half a unit: 2^-9 bf16, 2^-12 f16, of the largest value; twice that is allowed); the
gradients see the rounded output through delta = sum(out * dout), whose error is that rounding times |dout| summed over the
head (sqrt(64) at most): eight times the forward bound."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention
from oops_b200.attention.triangle.triangle_attention import layout_agnostic_kernels
from oops_b200.runtime import cabi

pytestmark = pytest.mark.gpu
ROUNDING = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols,heads,dim,bias_kind,mask_kind,layout",
                         [(3, 1, 2, 8, "none", "none", "plain"), (5, 63, 3, 1, "shared", "random", "plain"),
                          (40, 64, 2, 64, "shared", "ones", "plain"), (9, 65, 2, 40, "full", "tokens", "plain"),
                          (70, 130, 2, 24, "shared32", "tokens", "swapped"), (6, 200, 2, 48, "shared", "random", "head"),
                          (4, 97, 2, 33, "full32", "random", "swapped"), (8, 72, 2, 32, "shared", "random", "odd"),
                          (5, 136, 2, 32, "shared32", "none", "plain")])
def test_tile_edges(cuda, dtype, rows, cols, heads, dim, bias_kind, mask_kind, layout):
    gen = torch.Generator().manual_seed(cols)
    shape = (1, rows, cols, heads, dim)
    q, k, v = ((0.5 * torch.randn(shape, generator=gen)).to(dtype) for _ in range(3))
    up = torch.randn(shape, generator=gen).to(dtype)
    bias = None
    if bias_kind != "none":
        groups = 1 if bias_kind.startswith("shared") else rows
        bias = torch.randn(1, groups, heads, cols, cols, generator=gen).to(torch.float32 if bias_kind.endswith("32") else dtype)
    mask = {"none": None, "ones": torch.ones(1, rows, cols, dtype=torch.bool),
            "random": torch.rand(1, rows, cols, generator=gen) > 0.3,
            "tokens": ((torch.arange(cols) < max(1, cols // 2 - 3)) & (torch.arange(rows)[:, None] > 1))[None]}[mask_kind]
    if mask is not None:  # dropped keys may hold anything
        k, v = k.masked_fill(~mask[..., None, None], float("inf")), v.masked_fill(~mask[..., None, None], float("nan"))

    def laid_out(t):
        t = t.to(cuda)
        if layout == "swapped":
            t = t.transpose(1, 2).contiguous().transpose(1, 2)
        elif layout == "head":
            t = t.transpose(2, 3).contiguous().transpose(2, 3)
        elif layout == "odd":  # rows that start 2 bytes behind a 16-byte boundary
            t = torch.nn.functional.pad(t, (1, 0))[..., 1:]
        return t.detach().requires_grad_(True)

    leaves = [laid_out(t) for t in (q, k, v)] + ([] if bias is None else [bias.to(cuda).requires_grad_(True)])
    problem = cabi.make_problem(leaves[0].detach(), leaves[1].detach(), leaves[2].detach(), None,
                                None if bias is None else leaves[3].detach(), dim**-0.5)
    assert cabi.library().oops_ta_uses_tensor_path(cabi.byref(problem), 1) == 0
    out = triangle_attention(*leaves[:3], None if mask is None else mask.to(cuda), None if bias is None else leaves[3])
    grads = torch.autograd.grad(out, leaves, up.to(cuda))

    finite = [torch.nan_to_num(t.double(), nan=0.0, posinf=0.0) for t in (q, k, v)]
    ref = [t.requires_grad_(True) for t in finite] + ([] if bias is None else [bias.double().requires_grad_(True)])
    want = oracle.reference_dense(ref[0], ref[1], ref[2], mask, None if bias is None else ref[3], compute_dtype=torch.float64)
    want_grads = torch.autograd.grad(want, ref, up.double())
    for name, got, exact in zip(("out", "dq", "dk", "dv", "dbias"), (out, *grads), (want, *want_grads)):
        got, exact = got.detach().double().cpu(), exact.detach()
        bound = ROUNDING[dtype] * (1 if name == "out" else 8) * max(1.0, float(exact.abs().max()))
        error = float((got - exact).abs().max())
        assert error <= bound, (name, error, bound)
    if mask is not None:
        assert torch.count_nonzero(out.detach().cpu()[~mask.any(-1)]) == 0
        for grad in grads[1:3]:
            assert torch.count_nonzero(grad.cpu()[~mask]) == 0


@pytest.mark.parametrize("dtype,bias_dtype,low", [(torch.bfloat16, torch.bfloat16, -1e9), (torch.bfloat16, torch.bfloat16, None),
                                                  (torch.bfloat16, torch.float32, -1e9), (torch.float16, torch.float32, None),
                                                  (torch.float16, torch.float16, None)])
@pytest.mark.parametrize("dim", [24, 64])
def test_rows_under_a_low_bias(cuda, dtype, bias_dtype, low, dim):
    """Half of the queries have every key under a large negative bias (None: the lowest value of its type).  Their logits lose
    digits in f32 (all of them at -1e9, where the softmax is uniform); results and gradients are those that the
    layout-agnostic kernels take from the same f32 logits and lse.  Both paths round the result once; the gradients see it
    through delta (see the top of the file)."""
    gen = torch.Generator().manual_seed(dim)
    rows, cols, heads = 5, 70, 2
    q, k, v, up = (torch.randn(1, rows, cols, heads, dim, generator=gen).to(dtype).to(cuda) for _ in range(4))
    bias = torch.randn(1, 1, heads, cols, cols, generator=gen).to(bias_dtype)
    low = torch.finfo(bias_dtype).min if low is None else low
    bias[..., cols // 2:, :] = low

    def call():
        leaves = [t.detach().requires_grad_(True) for t in (q, k, v, bias.to(cuda))]
        out = triangle_attention(*leaves[:3], None, leaves[3])
        return [out.detach(), *torch.autograd.grad(out, leaves, up)]

    got = call()
    with layout_agnostic_kernels():
        want = call()
    for name, a, b in zip(("out", "dq", "dk", "dv", "dbias"), got, want):
        bound = 2 * ROUNDING[dtype] * (1 if name == "out" else 8) * max(1.0, float(b.double().abs().max()))
        assert float((a.double() - b.double()).abs().max()) <= bound, name
    if low < -2.0**29:
        uniform = v.double().mean(2, keepdim=True).expand(-1, -1, cols - cols // 2, -1, -1)
        assert float((got[0][:, :, cols // 2:].double() - uniform).abs().max()) <= ROUNDING[dtype] * float(v.double().abs().max())


@pytest.mark.parametrize("dim,cols", [(24, 70), (64, 64), (16, 130)])
@pytest.mark.parametrize("kind", ["scaled loss", "small gradients", "rising", "light keys"])
def test_f16_gradients_outside_the_range_of_f16(cuda, kind, dim, cols):
    """dS above 65504, dS below 2^-25, steps whose dS grows by 2^22 and more from one key or query tile to the next, and
    probabilities below 2^-25, each with results that f16 holds.  Bounds as at the top of the file, relative to the largest
    value of the result, and half a unit of the smallest f16 numbers (2^-25) on top."""
    gen = torch.Generator().manual_seed(dim)
    rows, heads = 2, 2
    shape = (1, rows, cols, heads, dim)
    q, k, v, up = (torch.randn(shape, generator=gen) for _ in range(4))
    bias = torch.randn(1, 1, heads, cols, cols, generator=gen)
    checked = (0, 1, 2, 3, 4)
    if kind == "scaled loss":  # dP = sum_d dO V is some 2^18 (its 2^-3 share still passes 65504), dQ and dK some 2^-8 of it
        up = 2.0**14 * (1 + 0.1 * up)
        v = torch.where(torch.rand(1, rows, cols, heads, 1, generator=gen) < 0.5, -1.0, 1.0) * (2 + 0.1 * v)
        q, k, bias = 2.0**-9 * q, 2.0**-9 * k, bias.clone()
        bias[..., :2] += 6  # two keys carry most of the weight
        checked = (1, 2)  # dV passes 65504 where it sums that upstream over all queries
    elif kind == "small gradients":
        up, k, q = 2.0**-16 * up, 512 * k, q / 512
    elif kind == "rising":
        behind = torch.arange(cols) // 64  # the first tile of keys weighs 2^-29, its queries get an upstream of 2^-14
        bias[..., behind == 0] -= 20.0 * int(behind.max())
        up = up * (2.0**-14 * 2.0 ** (22.0 * behind.clamp(max=1)))[:, None, None]
    else:
        bias[..., cols // 2:] -= 14
        up = 1000 * up
        checked = (3,)
    q, k, v, up, bias = (t.to(torch.float16) for t in (q, k, v, up, bias))
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v, bias)]
    out = triangle_attention(*leaves[:3], None, leaves[3])
    results = [out.detach(), *torch.autograd.grad(out, leaves, up.to(cuda))]
    ref = [t.double().requires_grad_(True) for t in (q, k, v, bias)]
    want = oracle.reference_dense(ref[0], ref[1], ref[2], None, ref[3], compute_dtype=torch.float64)
    wants = [want.detach(), *torch.autograd.grad(want, ref, up.double())]
    for i in checked:
        got, exact = results[i].double().cpu(), wants[i]
        if kind == "light keys":  # the gradient of the values behind the bias step, on its own scale
            got, exact = got[:, :, cols // 2:], exact[:, :, cols // 2:]
        largest = float(exact.abs().max())
        assert largest < 65504, (i, largest)
        bound = ROUNDING[torch.float16] * (1 if i == 0 else 8) * largest + 2.0**-25
        error = float((got - exact).abs().max())
        assert error <= bound, (("out", "dq", "dk", "dv", "dbias")[i], error, bound, largest)
