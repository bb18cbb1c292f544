"""Statistics warp of the single-pass reverse kernel: rows whose dots it makes itself (above 512 columns, one group of query tiles) and rows
whose dots a launch of their own makes, several items per CTA, ragged ends, outputs off 16-byte words, masks (prefixes, scattered keys,
the same keys in all rows that keep any, none) over dropped keys and values that are not finite.  16-bit bounds as in the parity tests: 2e-2 of the largest value
(at least 1); gradients of dropped keys and values are exactly zero."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention

pytestmark = pytest.mark.gpu


def _close(name, got, ref):
    error = float((got.detach().float().cpu() - ref).abs().max())
    assert error <= 2e-2 * max(1.0, float(ref.abs().max())), (name, error)


@pytest.mark.parametrize("kind", ["none", "prefix", "scattered", "tokens", "empty"])
@pytest.mark.parametrize("dtype,batch,rows,n,heads", [(torch.bfloat16, 1, 80, 129, 4), (torch.float16, 2, 80, 256, 2), (torch.bfloat16, 1, 64, 513, 3),
                                                      (torch.float16, 3, 64, 200, 1), (torch.bfloat16, 1, 64, 768, 3), (torch.bfloat16, 1, 64, 800, 1)])
def test_gradients(cuda, kind, dtype, batch, rows, n, heads):
    gen = torch.Generator().manual_seed(n)
    q, k, v, up = (torch.randn(batch, rows, n, heads, 32, generator=gen).to(dtype) for _ in range(4))
    bias = torch.randn(batch, 1, heads, n, n, generator=gen).to(dtype)
    mask = None
    if kind == "prefix":
        mask = torch.arange(n) < torch.randint(-n // 8, n + 1, (batch, rows, 1), generator=gen)
    elif kind == "scattered":
        mask = torch.rand(batch, rows, n, generator=gen) < 0.7
    elif kind == "tokens":  # every row of a sample that keeps a key keeps the same ones; whole key tiles are dropped
        ends = torch.tensor([n - n // 3, n // 2, n])[:batch, None, None]
        live = (torch.arange(rows) < rows - rows // 5) & (torch.arange(rows) != 3)
        mask = (torch.arange(n) < ends) & live[None, :, None]
    elif kind == "empty":
        mask = torch.zeros(batch, rows, n, dtype=torch.bool)
    want = oracle.forward_backward(q, k, v, mask, bias, up)
    if mask is not None:
        dead = ~mask[..., None, None]
        k, v = k.masked_fill(dead, float("inf")), v.masked_fill(dead, float("nan"))
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v, bias)]
    out = triangle_attention(*leaves[:3], None if mask is None else mask.to(cuda), leaves[3])
    grads = torch.autograd.grad(out, leaves, up.to(cuda))
    for name, got, ref in zip(("out", "dq", "dk", "dv", "dbias"), (out, *grads), want):
        _close(name, got, ref)
    if mask is not None:
        for got in grads[1:3]:
            assert not got.cpu()[~mask].any()


def test_output_off_words(cuda):
    """The C entry with an output whose rows are no 16-byte words: its dots are made by the launch that takes any stride."""
    from oops_b200.runtime import cabi

    gen = torch.Generator().manual_seed(3)
    rows, n, heads = 8, 600, 2
    q, k, v, up = (torch.randn(1, rows, n, heads, 32, generator=gen).to(torch.bfloat16) for _ in range(4))
    want = oracle.forward_backward(q, k, v, None, None, up)
    q, k, v, up = (t.to(cuda) for t in (q, k, v, up))
    lib, stream = cabi.library(), torch.cuda.current_stream().cuda_stream
    out = torch.empty(1, rows, n, heads, 33, dtype=torch.bfloat16, device=cuda)[..., :32]
    lse = torch.empty(rows * heads * n, device=cuda)
    problem = cabi.make_problem(q, k, v, None, None, 32**-0.5)
    pair = cabi.pair_of(out)
    assert lib.oops_ta_forward(cabi.byref(problem), cabi.byref(pair), lse.data_ptr(), stream) == 0
    grads = [torch.empty_like(q) for _ in range(3)]
    wanted = cabi.Grads()
    wanted.dq, wanted.dk, wanted.dv = (cabi.pair_of(g) for g in grads)
    scratch = torch.empty(int(lib.oops_ta_backward_workspace_bytes(cabi.byref(problem), cabi.byref(wanted))), dtype=torch.uint8, device=cuda)
    problem.workspace, problem.workspace_bytes = scratch.data_ptr(), scratch.numel()
    dout = cabi.pair_of(up)
    status = lib.oops_ta_backward(cabi.byref(problem), cabi.byref(pair), cabi.byref(dout), lse.data_ptr(), cabi.byref(wanted), stream)
    assert status == 0
    for name, got, ref in zip(("out", "dq", "dk", "dv"), (out, *grads), want):
        _close(name, got, ref)
