"""Which calls of the triangle multiplicative update take the fused passes and which are composed from single operations."""

import pytest
import torch

from oops_b200.pair.triangle_multiplication import _fused_serves


@pytest.mark.parametrize("shape,hidden,serves", [((65535, 16, 16, 8), 8, True), ((65536, 16, 16, 8), 8, False), ((256, 256, 16, 16, 8), 8, False),
                                                 ((46336, 46336, 1), 1, True), ((46344, 46344, 1), 1, False), ((46344, 46344, 1), 512, False),
                                                 ((16, 16, 8), 512, True), ((16, 16, 8), 513, False)])
def test_launch_limits(shape, hidden, serves):
    assert _fused_serves(torch.empty(shape, device="meta"), None, hidden, (), ()) is serves


@pytest.mark.parametrize("shape,serves", [((8,), True), ((1,), False), ((1, 8), False), ((7,), False), ((16, 8), False)])
def test_bias_shapes(shape, serves):
    projections = [torch.empty(8, 4) for _ in range(6)]
    biases = [None] * 5 + [torch.empty(shape)]
    assert _fused_serves(torch.empty(1, 16, 16, 4), None, 8, projections, biases) is serves


@pytest.mark.parametrize("dtype,prefix,tokens,serves", [(torch.bfloat16, 4096, 2, False), (torch.bfloat16, 4096, 6, False), (torch.bfloat16, 4096, 3, True),
                                                        (torch.bfloat16, 4096, 1, False), (torch.bfloat16, 4096, 8, True), (torch.bfloat16, 1024, 2, True),
                                                        (torch.float32, 4096, 4, False), (torch.float32, 4096, 5, True), (torch.float32, 16, 1, True)])
def test_many_grids_that_are_mostly_padding(dtype, prefix, tokens, serves):
    assert _fused_serves(torch.empty(prefix, tokens, tokens, 64, dtype=dtype, device="meta"), None, 64, (), ()) is serves


def test_subclasses_are_composed():
    class Labelled(torch.Tensor):
        pass

    plain = [torch.empty(8, 4) for _ in range(6)]
    pair = torch.empty(1, 16, 16, 4)
    assert _fused_serves(pair, None, 8, [torch.nn.Parameter(p) for p in plain], [None] * 6)
    assert not _fused_serves(pair.as_subclass(Labelled), None, 8, plain, [None] * 6)
    assert not _fused_serves(pair, None, 8, [*plain[:5], plain[5].as_subclass(Labelled)], [None] * 6)
