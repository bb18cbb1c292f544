"""Parameters of the multiplicative update's output norm that start off a 16-byte boundary, in channels on either side of a group of eight, give
what aligned copies of them give, bit for bit."""

import pytest
import torch

import oops_b200 as oops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,params,channels", [(torch.bfloat16, torch.float32, 64), (torch.float16, torch.float16, 40),
                                                   (torch.bfloat16, torch.bfloat16, 20), (torch.float32, torch.float32, 72)])
def test_unaligned(cuda, dtype, params, channels):
    gen = torch.Generator(device=cuda).manual_seed(channels)
    pair = torch.randn(1, 19, 19, channels, device=cuda, generator=gen).to(dtype)
    weights = {f"{which}_weight": (channels**-0.5 * torch.randn(channels, channels, device=cuda, generator=gen)).to(params)
               for which in ("left_value", "left_gate", "right_value", "right_gate", "output", "output_gate")}
    norms = {f"{which}_norm_{what}": torch.randn(channels + 1, device=cuda, generator=gen).to(params)[1:]
             for which in ("input", "output") for what in ("weight", "bias")}
    with torch.no_grad():
        got = oops.triangle_multiplication(pair, None, direction="outgoing", **weights, **norms)
        want = oops.triangle_multiplication(pair, None, direction="outgoing", **weights, **{k: v.clone() for k, v in norms.items()})
    assert torch.equal(got, want)
