"""The closed copy of a row-shared bias: what samples of one call it is made for, and that each of them then gets the right walk.  Samples that keep
everything, the same first keys, other keys in every row, and nothing, side by side in one call; more samples than a warp has lanes;
a bias as a projection leaves it.  16-bit bounds as in the parity tests: 2e-2 of the largest value (at least 1)."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention
from oops_b200.runtime import cabi

pytestmark = pytest.mark.gpu


def _mask(kind, rows, n, gen):
    keys, row = torch.arange(n), torch.arange(rows)[:, None]
    return {"ones": torch.ones(rows, n, dtype=torch.bool), "tokens": (keys < n - n // 3) & (row < rows - rows // 8),
            "scattered": torch.rand(rows, n, generator=gen) < 0.7, "nothing": torch.zeros(rows, n, dtype=torch.bool),
            "staircase": keys <= row * n // rows}[kind]


@pytest.mark.parametrize("kinds", [("ones", "tokens"), ("tokens", "scattered"), ("ones", "nothing"), ("nothing", "tokens", "ones"), ("ones", "staircase"),
                                   ("ones",) * 32 + ("tokens",)])
@pytest.mark.parametrize("n,permuted", [(256, False), (200, True), (399, False)])
def test_samples(cuda, kinds, n, permuted):
    gen = torch.Generator().manual_seed(n + len(kinds))
    batch, rows, heads = len(kinds), 64, 2
    if batch > 8:
        heads = 1
    if n > 384:  # the forward copy starts with these
        rows = 128 if batch < 8 else 64
    q, k, v, up = (torch.randn(batch, rows, n, heads, 32, generator=gen).to(torch.bfloat16) for _ in range(4))
    bias = torch.randn(batch, 1, heads, n, n, generator=gen).to(torch.bfloat16)
    mask = torch.stack([_mask(kind, rows, n, gen) for kind in kinds])
    want = oracle.forward_backward(q, k, v, mask, bias, up)
    dead = ~mask[..., None, None]
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k.masked_fill(dead, float("inf")), v.masked_fill(dead, float("nan")))]
    b = bias.to(cuda)
    if permuted:
        b = b.permute(0, 1, 3, 4, 2).contiguous().permute(0, 1, 4, 2, 3)
    leaves.append(b.requires_grad_(True))
    out = triangle_attention(*leaves[:3], mask.to(cuda), leaves[3])
    grads = torch.autograd.grad(out, leaves, up.to(cuda))
    for name, got, ref in zip(("out", "dq", "dk", "dv", "dbias"), (out, *grads), want):
        error = float((got.detach().float().cpu() - ref).abs().max())
        assert error <= 2e-2 * max(1.0, float(ref.abs().max())), (name, error)
    for got in grads[1:3]:
        assert not got.cpu()[~mask].any()


@pytest.mark.parametrize("kind,n,copied", [("ones", 256, False), ("scattered", 256, False), ("staircase", 256, False), ("scattered", 300, True),
                                           ("tokens", 256, True), ("tokens", 300, True), ("ones", 300, True)])
def test_reverse_copies_what_a_walk_needs(cuda, kind, n, copied):
    gen = torch.Generator().manual_seed(n)
    rows, heads, row = 64, 2, (n + 127) // 128 * 128
    q, k, v, up = (torch.randn(1, rows, n, heads, 32, generator=gen).to(cuda, torch.bfloat16) for _ in range(4))
    bias = torch.randn(1, 1, heads, n, row, generator=gen).to(cuda, torch.bfloat16)[..., :n]
    mask = _mask(kind, rows, n, gen)[None].to(cuda)
    lib, stream = cabi.library(), torch.cuda.current_stream().cuda_stream
    out, lse = torch.empty_like(q), torch.empty(rows * heads * n, device=cuda)
    problem, pair, dout = cabi.make_problem(q, k, v, mask, bias, 32**-0.5), cabi.pair_of(out), cabi.pair_of(up)
    assert lib.oops_ta_forward(cabi.byref(problem), cabi.byref(pair), lse.data_ptr(), stream) == 0
    grads, (dq, dk, dv) = cabi.Grads(), (torch.empty_like(q) for _ in range(3))
    grads.dq, grads.dk, grads.dv = cabi.pair_of(dq), cabi.pair_of(dk), cabi.pair_of(dv)
    scratch = torch.full((int(lib.oops_ta_backward_workspace_bytes(cabi.byref(problem), cabi.byref(grads))),), 77, dtype=torch.uint8, device=cuda)
    problem.workspace, problem.workspace_bytes = scratch.data_ptr(), scratch.numel()
    assert lib.oops_ta_backward(cabi.byref(problem), cabi.byref(pair), cabi.byref(dout), lse.data_ptr(), cabi.byref(grads), stream) == 0
    assert bool((scratch[-heads * n * row * 2:] != 77).any()) == copied
