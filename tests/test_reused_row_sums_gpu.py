"""A reverse pass in two calls, the second of which finds the row sums of the first in its workspace: they are all it may rely on
there, so the rest of the workspace is filled with noise in between."""

import pytest
import torch

from oops_b200.attention.triangle import function as fn
from oops_b200.runtime import cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,cols", [(32, 136), (32, 256), (24, 70)])
@pytest.mark.parametrize("mask_kind", ["none", "ones", "tokens", "random"])
def test_second_call(cuda, dim, cols, mask_kind):
    gen = torch.Generator().manual_seed(cols)
    rows, heads = 20, 2
    q, k, v, up = (torch.randn(1, rows, cols, heads, dim, generator=gen).to(cuda, torch.bfloat16) for _ in range(4))
    bias = torch.randn(1, 1, heads, cols, cols, generator=gen).to(cuda, torch.bfloat16)
    mask = {"none": None, "ones": torch.ones(1, rows, cols, dtype=torch.bool),
            "tokens": (torch.arange(cols) < cols - 30).expand(1, rows, cols).contiguous(),
            "random": torch.rand(1, rows, cols, generator=gen) > 0.3}[mask_kind]
    mask = None if mask is None else mask.to(cuda)
    geometry, scale = fn.DenseGeometry(), dim**-0.5
    out, lse = fn.run_forward(geometry, q, k, v, mask, bias, scale, 0, True)
    wants = ((False, False, False, True), (True, True, True, False))
    scratch = torch.empty(max(fn.backward_scratch_bytes(q, k, v, mask, bias, scale, 0, w) for w in wants), dtype=torch.uint8, device=cuda)

    def call(want, flags):
        got = fn.run_backward(geometry, up, q, k, v, mask, bias, out, lse, scale, flags, want, scratch=scratch)
        return [g for g in got if g is not None]

    fresh = [call(w, 0) for w in wants]
    call(wants[0], 0)
    for want, expected in zip(wants, fresh):
        scratch[4 * rows * heads * cols:].random_(0, 256)
        for got, exact in zip(call(want, cabi.FLAG_REUSE_DELTA), expected):
            assert torch.equal(got, exact)
