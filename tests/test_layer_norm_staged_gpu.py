"""Layer norm on rows that travel through shared memory a turn ahead: row counts on either side of a turn of a warp and of all of them, widths on
either side of the lane groups that share a row, strided rows, gradients wanted in part; against f64.  The norm of a 16-bit result's error
is that of its rounding (half a unit at most: 2^-9 bf16, 2^-12 f16 of the values); f32 sums of up to 512 terms are off by some
units of 2^-24 (the parameters' gradients by those of a sum over the rows)."""

import pytest
import torch

import oops_b200 as oops

pytestmark = pytest.mark.gpu
ROUNDING = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11, torch.float32: 1e-6}


@pytest.mark.parametrize("dtype,rows,width,stride", [(torch.bfloat16, 1, 128, 0), (torch.float16, 9, 8, 0), (torch.bfloat16, 4737, 72, 0),
                                                     (torch.bfloat16, 19000, 128, 136), (torch.float16, 4735, 200, 0),
                                                     (torch.bfloat16, 2371, 264, 520), (torch.float32, 33, 4, 0), (torch.float32, 9473, 68, 0),
                                                     (torch.float32, 7105, 128, 132), (torch.float32, 2369, 256, 0)])
def test_edges(cuda, dtype, rows, width, stride):
    gen = torch.Generator(device=cuda).manual_seed(rows)
    storage = torch.randn(rows, stride or width, device=cuda, generator=gen).to(dtype)
    x = storage[:, :width].detach().requires_grad_(True)
    w, b = (torch.randn(width, device=cuda, generator=gen).requires_grad_(True) for _ in range(2))
    up = torch.randn(rows, width, device=cuda, generator=gen).to(dtype)
    y = oops.layer_norm(x, width, w, b)
    grads = torch.autograd.grad(y, (x, w, b), up, retain_graph=True)
    exact = [t.detach().double().requires_grad_(True) for t in (x, w, b)]
    want = torch.nn.functional.layer_norm(exact[0], (width,), exact[1], exact[2])
    for name, got, ref in zip(("y", "dx", "dw", "db"), (y, *grads), (want, *torch.autograd.grad(want, exact, up.double()))):
        bound = ROUNDING[dtype if name in ("y", "dx") else torch.float32]
        assert float((got.detach().double() - ref).norm()) <= bound * max(float(ref.norm()), 1e-3), name
    dw, = torch.autograd.grad(y, (w,), up)
    assert torch.equal(dw, grads[1])


@pytest.mark.parametrize("width,turns,short", [(128, 1, 0), (128, 2, 0), (128, 2, 3), (64, 2, 0), (256, 2, 1), (512, 2, 0), (128, 3, 0), (128, 1, 9000)])
def test_parameter_gradients_after_the_last_request(cuda, width, turns, short):
    """The sums of the parameters' gradients take the shared memory that the request for a turn behind the last one writes zeros to: row counts
    of an even and an odd number of turns, and warps that have none.  The sums have an order, so that all repetitions agree."""
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    lanes = 8 if width <= 64 else 16 if width <= 128 else 32
    rows = sms * 2 * 8 * (4 // (2 * max(1, width // 256))) * (32 // lanes) * turns - short  # CTAs, warps, row blocks of a turn, rows of a block
    gen = torch.Generator(device=cuda).manual_seed(width + turns)
    x = torch.randn(rows, width, device=cuda, generator=gen).bfloat16()
    up = torch.randn(rows, width, device=cuda, generator=gen).bfloat16()
    w, b = (torch.randn(width, device=cuda, generator=gen).requires_grad_(True) for _ in range(2))
    y = oops.layer_norm(x, width, w, b)
    first = torch.autograd.grad(y, (w, b), up, retain_graph=True)
    for _ in range(50):
        assert all(torch.equal(p, q) for p, q in zip(torch.autograd.grad(y, (w, b), up, retain_graph=True), first))
    exact = [t.detach().double().requires_grad_(True) for t in (x, w, b)]
    want = torch.autograd.grad(torch.nn.functional.layer_norm(exact[0], (width,), exact[1], exact[2]), exact[1:], up.double())
    for got, ref in zip(first, want):
        assert float((got.double() - ref).norm()) <= ROUNDING[torch.float32] * float(ref.norm())


@pytest.mark.parametrize("dtype,width", [(torch.bfloat16, 128), (torch.float16, 384), (torch.float32, 384), (torch.float32, 64)])
@pytest.mark.parametrize("share,off", [(1, 0), (1, 1), (2, 0), (2, 1), (3, 1), (4, -1)])
def test_shares_of_a_turn(cuda, dtype, width, share, off):
    """Fewer row blocks than a turn of one CTA per SM: row counts on either side of one, two, three and four blocks a warp."""
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    units = width * dtype.itemsize // 16
    rows = sms * 8 * share * (4 if units <= 8 else 2 if units <= 16 else 1) + off
    gen = torch.Generator(device=cuda).manual_seed(rows)
    x, up = (torch.randn(rows, width, device=cuda, generator=gen).to(dtype) for _ in range(2))
    leaves = [x.requires_grad_(True)] + [torch.randn(width, device=cuda, generator=gen).requires_grad_(True) for _ in range(2)]
    y = oops.layer_norm(leaves[0], width, leaves[1], leaves[2])
    exact = [t.detach().double().requires_grad_(True) for t in leaves]
    want = torch.nn.functional.layer_norm(exact[0], (width,), exact[1], exact[2])
    for name, got, ref in zip(("y", "dx", "dw", "db"), (y, *torch.autograd.grad(y, leaves, up)), (want, *torch.autograd.grad(want, exact, up.double()))):
        bound = ROUNDING[dtype if name in ("y", "dx") else torch.float32]
        assert float((got.detach().double() - ref).norm()) <= bound * float(ref.norm()), name
