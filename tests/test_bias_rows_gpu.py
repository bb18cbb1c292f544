"""The bias rows of the TMA kernels: any strides in, whole 16-byte words out, bytes unchanged; and the gradient that comes back."""

import ctypes

import pytest
import torch

from oops_b200 import triangle_attention
from oops_b200.runtime import cabi

pytestmark = pytest.mark.gpu


def _bias(n, layout, dtype, device, groups=1):
    gen = torch.Generator().manual_seed(n)
    if layout == "projected":  # as a linear map over the pair leaves it: heads innermost
        return torch.randn(2, groups, n, n, 3, generator=gen).to(device, dtype).permute(0, 1, 4, 2, 3)
    if layout == "transposed":
        return torch.randn(2, groups, 3, n, n, generator=gen).to(device, dtype).transpose(-1, -2)
    return torch.randn(2, groups, 3, n, n, generator=gen).to(device, dtype)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 100, 131, 264])
@pytest.mark.parametrize("layout,groups", [("contiguous", 1), ("projected", 1), ("transposed", 2)])
def test_bytes(cuda, n, layout, groups):
    bias = _bias(n, layout, torch.bfloat16, cuda, groups)
    row = (n + 7) // 8 * 8
    rows = torch.full((2, groups, 3, n, row), float("nan"), dtype=torch.bfloat16, device=cuda)
    strides = (ctypes.c_int64 * 5)(*bias.stride())
    stream = torch.cuda.current_stream(cuda).cuda_stream
    assert cabi.library().oops_ta_bias_rows(2, groups, 3, n, ctypes.c_void_p(bias.data_ptr()), strides, ctypes.c_void_p(rows.data_ptr()),
                                            ctypes.c_void_p(stream)) == 0
    assert torch.equal(rows[..., :n].view(torch.int16), bias.contiguous().view(torch.int16))
    assert torch.count_nonzero(rows[..., n:]) == 0


@pytest.mark.parametrize("n,layout", [(100, "projected"), (104, "projected"), (65, "contiguous")])
def test_gradient_keeps_its_place(cuda, n, layout):
    gen = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(2, n, n, 3, 32, generator=gen).to(cuda, torch.bfloat16) for _ in range(3))
    bias = _bias(n, layout, torch.bfloat16, cuda).requires_grad_(True)
    padded = torch.nn.functional.pad(bias.detach(), (0, -n % 8)).contiguous()[..., :n].requires_grad_(True)
    up = torch.randn(q.shape, generator=gen).to(cuda, torch.bfloat16)
    results = [torch.autograd.grad(triangle_attention(q, k, v, None, b), b, up)[0] for b in (bias, padded)]
    assert results[0].shape == bias.shape and torch.equal(*results)


def test_more_words_than_32_bits_count(cuda):
    """2^32 words: one plane of 16384 x 16384 values seen by 128 heads."""
    torch.cuda.empty_cache()
    heads, n = 128, 16384
    if torch.cuda.mem_get_info(cuda)[0] < heads * n * n * 2 + (8 << 30):
        pytest.skip("needs 72 GB of device memory")
    plane = torch.randint(-(2**15), 2**15, (n, n), dtype=torch.int16, device=cuda)
    rows = torch.empty(heads, n, n, dtype=torch.int16, device=cuda)
    rows[-1, -1].fill_(-1)
    stream = torch.cuda.current_stream(cuda).cuda_stream
    assert cabi.library().oops_ta_bias_rows(1, 1, heads, n, ctypes.c_void_p(plane.data_ptr()), (ctypes.c_int64 * 5)(0, 0, 0, n, 1),
                                            ctypes.c_void_p(rows.data_ptr()), ctypes.c_void_p(stream)) == 0
    for head in (0, 63, 127):
        assert torch.equal(rows[head], plane)
    del rows
    torch.cuda.empty_cache()
