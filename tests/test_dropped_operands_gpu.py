"""Token masks over operands that are not finite, in the reverse pass: infinities and NaN in the queries, keys, values and upstream gradients
of rows that keep no key, in dropped keys and values, and in the bias of a sample that keeps nothing, reach no gradient; a query or upstream
gradient of a row that keeps keys reaches none of its dropped keys.  Rows of one and of several groups of query tiles, with and without a
ragged key tile.  16-bit bounds as in the parity tests: 2e-2 of the largest value (at least 1)."""

import pytest
import torch

from oracle import triangle_oracle as oracle
from oops_b200 import triangle_attention

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")


def _gradients(cuda, q, k, v, mask, bias, up):
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v, bias)]
    out = triangle_attention(*leaves[:3], mask.to(cuda), leaves[3])
    return [t.detach().cpu() for t in (out, *torch.autograd.grad(out, leaves, up.to(cuda)))]


@pytest.mark.parametrize("dtype,batch,rows,n", [(torch.bfloat16, 1, 64, 192), (torch.float16, 2, 70, 256), (torch.bfloat16, 1, 64, 700),
                                                (torch.bfloat16, 1, 64, 800)])
def test_rows_that_keep_nothing(cuda, dtype, batch, rows, n):
    gen = torch.Generator().manual_seed(n)
    q, k, v, up = (torch.randn(batch, rows, n, 2, 32, generator=gen).to(dtype) for _ in range(4))
    bias = torch.randn(batch, 1, 2, n, n, generator=gen).to(dtype)
    live = torch.arange(rows) < rows - rows // 4
    mask = ((torch.arange(n) < n - n // 5) & live[:, None])[None].repeat(batch, 1, 1)
    if batch > 1:
        mask[1] = False
    want = oracle.forward_backward(q, k, v, mask, bias, up)
    if batch > 1:
        bias[1, ..., ::3], bias[1, ..., 1::3] = INF, NAN
    for row in range(rows):
        for b in range(batch):
            if not mask[b, row].any():
                q[b, row, ::2], q[b, row, 1::2] = INF, NAN
                up[b, row, ::3], up[b, row, 1::3] = NAN, -INF
    dead = ~mask[..., None, None]
    got = _gradients(cuda, q, k.masked_fill(dead, INF), v.masked_fill(dead, NAN), mask, bias, up)
    for name, g, ref in zip(("out", "dq", "dk", "dv", "dbias"), got, want):
        error = float((g.float() - ref).abs().max())
        assert error <= 2e-2 * max(1.0, float(ref.abs().max())), (name, error)
    for g in got[:2]:
        assert not g[~mask.any(-1)].any()
    for g in got[2:4]:
        assert not g[~mask].any()


@pytest.mark.parametrize("n", [256, 700, 800])
def test_dropped_keys_of_other_rows(cuda, n):
    gen = torch.Generator().manual_seed(n)
    rows = 64
    q, k, v, up = (torch.randn(1, rows, n, 1, 32, generator=gen).to(torch.bfloat16) for _ in range(4))
    bias = torch.randn(1, 1, 1, n, n, generator=gen).to(torch.bfloat16)
    mask = (torch.arange(n) < n - 70).expand(1, rows, n).contiguous()
    q[0, 3, 5], q[0, 4, 6, 0, 7], up[0, 5, 7] = NAN, INF, -INF
    got = _gradients(cuda, q, k, v, mask, bias, up)
    for g in got[2:4]:
        assert not g[~mask].any()
    fine = torch.ones(rows, dtype=torch.bool)
    fine[3:6] = False
    for g in got[:4]:
        assert torch.isfinite(g[0, fine]).all()


@pytest.mark.parametrize("rows,n,masked", [(128, 390, False), (128, 447, False), (2, 700, False), (64, 700, False), (64, 1000, False),
                                           (64, 256, True), (64, 700, True), (64, 800, True)])
def test_rows_whose_logits_are_minus_infinity(cuda, rows, n, masked):
    """A query that holds an infinity and whose products with the kept keys are minus infinity, all of them, has no probability: zeros."""
    gen = torch.Generator().manual_seed(n)
    q, k, v, up = (torch.randn(1, rows, n, 1, 32, generator=gen).to(torch.bfloat16) for _ in range(4))
    bias = torch.randn(1, 1, 1, n, n, generator=gen).to(torch.bfloat16)
    mask = torch.ones(1, rows, n, dtype=torch.bool)
    if masked:
        mask[..., n - 70:] = False
    k[0, 1, :, 0, 9] = -k[0, 1, :, 0, 9].abs() - 1.0
    empty = [n // 2, n - 1, 3]
    q[0, 1, empty, 0, 9] = INF
    q[0, 0, 6, 0, 9] = INF  # (its keys have both signs: NaN)
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v, bias)]
    out = triangle_attention(*leaves[:3], mask.to(cuda) if masked else None, leaves[3])
    dq, dk, dv, _ = torch.autograd.grad(out, leaves, up.to(cuda))
    for got in (out, dq):
        assert not got[0, 1, empty].any()
        assert torch.isnan(got[0, 0, 6]).all()
        got = got.detach().clone()
        got[0, 0, 6] = 0
        assert torch.isfinite(got).all()
    assert torch.isfinite(dv[0, 1:]).all()


@pytest.mark.parametrize("rows,n", [(128, 399), (160, 450), (128, 700)])
def test_gated_rows_whose_logits_are_minus_infinity(cuda, rows, n):
    """The same through the gated form, whose gate then holds a NaN or none; one item a CTA and several."""
    from oops_b200 import triangle_attention_gated

    gen = torch.Generator().manual_seed(n)
    q, k, v, gate = (torch.randn(1, rows, n, 4, 32, generator=gen).to(torch.float16) for _ in range(4))
    bias = torch.randn(1, 1, 4, n, n, generator=gen).to(torch.float16)
    k[0, 1, :, 2, 9] = -k[0, 1, :, 2, 9].abs() - 1.0
    empty = [n // 2, n - 1, 3]
    q[0, 1, empty, 2, 9] = INF
    gate[0, 1, 3, 2, 5] = NAN
    with torch.no_grad():
        out = triangle_attention_gated(*(t.to(cuda) for t in (q, k, v, gate)), None, bias.to(cuda)).cpu()
    assert bool(torch.isnan(out[0, 1, 3, 2, 5]))
    out[0, 1, 3, 2, 5] = 0
    assert not out[0, 1, empty, 2].any()
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("rows,n,pad", [(64, 200, 20), (128, 399, 130), (64, 700, 60), (64, 801, 100)])
def test_padding_through_the_bias(cuda, rows, n, pad):
    """Padded queries and keys under a bias of minus infinity, without a mask: what the call without them gives, and zeros."""
    gen = torch.Generator().manual_seed(n)
    q, k, v, up = (torch.randn(1, rows, n, 2, 32, generator=gen).to(torch.bfloat16) for _ in range(4))
    bias = torch.randn(1, 1, 2, n, n, generator=gen).to(torch.bfloat16)
    kept = n - pad
    want = oracle.forward_backward(*(t[:, :, :kept] for t in (q, k, v)), None, bias[..., :kept, :kept], up[:, :, :kept])
    bias[..., kept:, :], bias[..., kept:] = -INF, -INF
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v, bias)]
    out = triangle_attention(*leaves[:3], None, leaves[3])
    got = [t.detach().float().cpu() for t in (out, *torch.autograd.grad(out, leaves, up.to(cuda)))]
    for name, g, ref in zip(("out", "dq", "dk", "dv"), got, want):
        error = float((g[:, :, :kept] - ref).abs().max())
        assert error <= 2e-2 * max(1.0, float(ref.abs().max())), (name, error)
        assert not g[:, :, kept:].any(), name
    error = float((got[4][..., :kept, :kept] - want[4]).abs().max())
    assert error <= 2e-2 * max(1.0, float(want[4].abs().max())), error
