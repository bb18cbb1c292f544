"""Row sums that the single-pass reverse kernel makes itself (513 to 768 columns, eight items a CTA and more): the gradients against the
oracle, for outputs on and off 16-byte words; and row sums of either origin found again by a second call, over masks and rows that the kernel has
walks of their own for.  16-bit bounds as in the parity tests: 2e-2 of the largest value (at least 1)."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200.attention.triangle import function as fn
from oops_b200.runtime import cabi

pytestmark = pytest.mark.gpu


def _many(n):
    """Rows of 16 heads that make eight items and more of every CTA."""
    return 8 * torch.cuda.get_device_properties(0).multi_processor_count // 16 + 1, n, 16


@pytest.mark.parametrize("dtype,n,wide", [(torch.bfloat16, 513, 32), (torch.float16, 768, 32), (torch.bfloat16, 600, 33)])
def test_gradients(cuda, dtype, n, wide):
    gen = torch.Generator().manual_seed(n)
    rows, n, heads = _many(n)
    q, k, v, up = (torch.randn(1, rows, n, heads, 32, generator=gen).to(cuda, dtype) for _ in range(4))
    lib, stream = cabi.library(), torch.cuda.current_stream().cuda_stream
    out = torch.empty(1, rows, n, heads, wide, dtype=dtype, device=cuda)[..., :32]
    lse = torch.empty(rows * heads * n, device=cuda)
    problem, pair, dout = cabi.make_problem(q, k, v, None, None, 32**-0.5), cabi.pair_of(out), cabi.pair_of(up)
    assert lib.oops_ta_forward(cabi.byref(problem), cabi.byref(pair), lse.data_ptr(), stream) == 0
    got, wanted = [torch.empty_like(q) for _ in range(3)], cabi.Grads()
    wanted.dq, wanted.dk, wanted.dv = (cabi.pair_of(g) for g in got)
    scratch = torch.empty(int(lib.oops_ta_backward_workspace_bytes(cabi.byref(problem), cabi.byref(wanted))), dtype=torch.uint8, device=cuda)
    problem.workspace, problem.workspace_bytes = scratch.data_ptr(), scratch.numel()
    assert lib.oops_ta_backward(cabi.byref(problem), cabi.byref(pair), cabi.byref(dout), lse.data_ptr(), cabi.byref(wanted), stream) == 0
    sums = (out.float() * up.float()).sum(-1).transpose(2, 3).reshape(-1)
    left = scratch[: 4 * rows * heads * n].view(torch.float32)
    assert float((left - sums).abs().max()) <= 1e-5 * float((out.float() * up.float()).abs().sum(-1).max())  # 32 products, at most 32 roundings of 2^-24 on each side
    picked = [0, rows // 2, rows - 1]  # rows are independent problems
    want = oracle.forward_backward(*(t[:, picked].cpu() for t in (q, k, v)), None, None, up[:, picked].cpu())
    for name, g, ref in zip(("out", "dq", "dk", "dv"), (out, *got), want):
        error = float((g[:, picked].float().cpu() - ref).abs().max())
        assert error <= 2e-2 * max(1.0, float(ref.abs().max())), (name, error)


@pytest.mark.parametrize("first", [0, 1])
@pytest.mark.parametrize("mask_kind", ["none", "ones", "tokens", "random"])
@pytest.mark.parametrize("cols,many", [(256, False), (700, False), (700, True), (800, False)])
def test_second_call(cuda, cols, many, mask_kind, first):
    """As in the test of reused row sums: they are all that a second call may rely on in the workspace."""
    gen = torch.Generator(device=cuda).manual_seed(cols)
    rows, cols, heads = _many(cols) if many else (64, cols, 2)
    q, k, v, up = (torch.randn(1, rows, cols, heads, 32, generator=gen, device=cuda).to(torch.bfloat16) for _ in range(4))
    bias = torch.randn(1, 1, heads, cols, (cols + 7) // 8 * 8, generator=gen, device=cuda).to(torch.bfloat16)[..., :cols]
    mask = {"none": None, "ones": torch.ones(1, rows, cols, dtype=torch.bool, device=cuda),
            "tokens": ((torch.arange(cols, device=cuda) < cols - 30) & (torch.arange(rows, device=cuda)[:, None] < rows - 5))[None],
            "random": torch.rand(1, rows, cols, generator=gen, device=cuda) > 0.3}[mask_kind]
    geometry, scale = fn.DenseGeometry(), 32**-0.5
    out, lse = fn.run_forward(geometry, q, k, v, mask, bias, scale, 0, True)
    wants = ((True, True, True, False), (False, False, False, True))
    scratch = torch.empty(max(fn.backward_scratch_bytes(q, k, v, mask, bias, scale, 0, w) for w in wants), dtype=torch.uint8, device=cuda)

    def call(want, flags):
        return [g for g in fn.run_backward(geometry, up, q, k, v, mask, bias, out, lse, scale, flags, want, scratch=scratch) if g is not None]

    fresh = [call(w, 0) for w in wants]
    call(wants[first], 0)
    for want, expected in zip(wants, fresh):
        scratch[4 * rows * heads * cols:].random_(0, 256)
        for got, exact in zip(call(want, cabi.FLAG_REUSE_DELTA), expected):
            assert torch.equal(got, exact)
