"""Ragged rows over a row-shared bias, which is closed with minus infinity in scratch: a few keys or nearly a whole tile behind the last step,
biases of several samples, permuted and with entries of minus infinity or far below zero, with and without a mask, and a caller whose
scratch has no room for the copy.  16-bit bounds as in the parity tests: 2e-2 of the largest value (at least 1)."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention
from oops_b200.runtime import cabi

pytestmark = pytest.mark.gpu


def _close(name, got, ref):
    error = float((got.detach().float().cpu() - ref).abs().max())
    assert error <= 2e-2 * max(1.0, float(ref.abs().max())), (name, error)


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("dtype,batch,rows,n,heads,bias_kind", [(torch.bfloat16, 1, 130, 385, 2, "plain"), (torch.float16, 2, 64, 200, 2, "permuted"),
                                                                (torch.bfloat16, 1, 129, 447, 1, "infinite"), (torch.float16, 1, 128, 390, 1, "low"),
                                                                (torch.bfloat16, 1, 64, 769, 1, "plain")])
def test_ragged(cuda, masked, dtype, batch, rows, n, heads, bias_kind):
    gen = torch.Generator().manual_seed(n)
    q, k, v, up = (torch.randn(batch, rows, n, heads, 32, generator=gen).to(dtype) for _ in range(4))
    bias = torch.randn(batch, 1, heads, n, n, generator=gen)
    if bias_kind == "permuted":
        bias = bias.permute(0, 1, 3, 4, 2).contiguous().permute(0, 1, 4, 2, 3)
    elif bias_kind == "infinite":
        bias[..., 1::3] = -float("inf")
    elif bias_kind == "low":  # every probability of a key behind the end would leave the range of 16 bits
        bias -= 40.0
    bias = bias.to(dtype)
    mask = torch.rand(batch, rows, n, generator=gen) < 0.8 if masked else None
    want = oracle.forward_backward(q, k, v, mask, bias, up)
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v, bias)]
    out = triangle_attention(*leaves[:3], None if mask is None else mask.to(cuda), leaves[3])
    grads = torch.autograd.grad(out, leaves, up.to(cuda))
    for name, got, ref in zip(("out", "dq", "dk", "dv", "dbias"), (out, *grads), want):
        _close(name, got, ref)


def test_scratch_without_room(cuda):
    gen = torch.Generator().manual_seed(5)
    rows, n, heads = 128, 401, 1
    q, k, v, up = (torch.randn(1, rows, n, heads, 32, generator=gen).to(cuda, torch.bfloat16) for _ in range(4))
    bias = torch.randn(1, 1, heads, n, (n + 7) // 8 * 8, generator=gen).to(cuda, torch.bfloat16)[..., :n]
    lib, stream = cabi.library(), torch.cuda.current_stream().cuda_stream
    results = []
    for room in (True, False):
        problem = cabi.make_problem(q, k, v, None, bias, 32**-0.5)
        need = int(lib.oops_ta_forward_workspace_bytes(cabi.byref(problem)))
        assert need > 0
        scratch = torch.empty(need, dtype=torch.uint8, device=cuda)
        if room:
            problem.workspace, problem.workspace_bytes = scratch.data_ptr(), need
        out, lse = torch.empty_like(q), torch.empty(rows * heads * n, device=cuda)
        pair = cabi.pair_of(out)
        assert lib.oops_ta_forward(cabi.byref(problem), cabi.byref(pair), lse.data_ptr(), stream) == 0
        grads = cabi.Grads()
        dq, dk, dv = (torch.empty_like(q) for _ in range(3))
        grads.dq, grads.dk, grads.dv = cabi.pair_of(dq), cabi.pair_of(dk), cabi.pair_of(dv)
        need = int(lib.oops_ta_backward_workspace_bytes(cabi.byref(problem), cabi.byref(grads)))
        less = need - heads * n * 512 * 2  # a row of whole key tiles has 512 elements
        scratch = torch.empty(need, dtype=torch.uint8, device=cuda)
        problem.workspace, problem.workspace_bytes = scratch.data_ptr(), need if room else less
        dout = cabi.pair_of(up)
        assert lib.oops_ta_backward(cabi.byref(problem), cabi.byref(pair), cabi.byref(dout), lse.data_ptr(), cabi.byref(grads), stream) == 0
        results.append((out, lse, dq, dk, dv))
    for a, b in zip(*results):
        assert torch.equal(a, b)
