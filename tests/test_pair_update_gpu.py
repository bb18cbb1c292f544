"""The passes of the triangle multiplicative update between its GEMMs at the sizes where their tiles end: one token, odd
token counts (padded planes), channel counts that are no multiple of 8 or 32, several prefix elements; against the oracle
in f64.  f32: the longest sum has tokens + channels terms, each product rounded once (2^-24), so 2e-5 of the largest value
is tens of roundings; 16-bit: every stage rounds its result once (2^-9 bf16, 2^-12 f16) and a gradient passes at most ten
stages whose roundings add up in the worst case."""

import pytest
import torch

import oops_b200 as oops
from oracle import triangle_multiplication_oracle as oracle
from test_triangle_multiplication_gpu import _weights

pytestmark = pytest.mark.gpu
TOL = {torch.float32: 2e-5, torch.float16: 10 * 2.0**-11, torch.bfloat16: 10 * 2.0**-8}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("prefix,tokens,channels,hidden,direction,masked",
                         [((), 1, 8, 8, "outgoing", False), ((2,), 7, 5, 3, "incoming", True), ((1,), 33, 40, 36, "outgoing", True),
                          ((3,), 17, 64, 200, "incoming", False), ((1,), 64, 128, 512, "outgoing", True)])
def test_tile_edges(dtype, prefix, tokens, channels, hidden, direction, masked):
    dev = torch.device("cuda", 0)
    gen = torch.Generator().manual_seed(tokens)
    shape = (*prefix, tokens, tokens, channels)
    pair, up = torch.randn(shape, generator=gen).to(dtype), torch.randn(shape, generator=gen).to(dtype)
    mask = torch.rand(shape[:-1], generator=gen).to(dtype) if masked else None
    weights = _weights(gen, channels, hidden, masked)
    leaves = [pair.to(dev).requires_grad_(True)] + [w.to(dev).requires_grad_(True) for w in weights.values()]
    out = oops.triangle_multiplication(leaves[0], None if mask is None else mask.to(dev), direction=direction,
                                       **dict(zip(weights, leaves[1:])))
    grads = torch.autograd.grad(out, leaves, up.to(dev))
    # the oracle sees the parameters as the 16-bit products do: projections rounded to the activation type
    rounded = {k: (w if "norm" in k else w.to(dtype)).double().requires_grad_(True) for k, w in weights.items()}
    pair_r = pair.double().requires_grad_(True)
    want = oracle.triangle_multiplication(pair_r, mask, direction=direction, dtype=torch.float64, **rounded)
    want_grads = torch.autograd.grad(want, [pair_r, *rounded.values()], up.double())
    for name, got, ref in zip(["out", "pair", *weights], [out, *grads], [want, *want_grads]):
        # one token normalises a rank-one update: its gradients are differences of equal terms, judged absolutely
        bound = TOL[dtype] * max(1.0, float(ref.detach().abs().max()))
        assert float((got.detach().double().cpu() - ref.detach()).abs().max()) <= bound, name


def test_more_prefix_elements_than_a_grid_axis_holds(cuda):
    gen = torch.Generator().manual_seed(7)
    weights = {k: w.to(cuda) for k, w in _weights(gen, 8, 8, True).items()}
    pair = torch.randn(65537, 9, 9, 8, generator=gen).to(cuda).requires_grad_(True)
    out = oops.triangle_multiplication(pair, **weights)
    (grad,) = torch.autograd.grad(out.sum(), pair)
    for part in (slice(0, 3), slice(65530, 65537)):
        piece = pair.detach()[part].requires_grad_(True)
        want = oops.triangle_multiplication(piece, **weights)
        (want_grad,) = torch.autograd.grad(want.sum(), piece)
        for got, exact in ((out.detach()[part], want.detach()), (grad[part], want_grad)):
            assert float((got - exact).abs().max()) <= TOL[torch.float32] * max(1.0, float(exact.abs().max()))


@pytest.mark.parametrize("name,rows", [("left_gate_bias", 24), ("output_bias", 16), ("output_gate_bias", 16)])
def test_projection_biases_that_broadcast(cuda, name, rows):
    gen = torch.Generator().manual_seed(8)
    weights = {k: w.to(cuda) for k, w in _weights(gen, 16, 24, False).items()}
    pair, value = torch.randn(1, 12, 12, 16, generator=gen).to(cuda), torch.randn(1, generator=gen).to(cuda)
    want = oops.triangle_multiplication(pair, **weights, **{name: value.expand(rows).contiguous()})
    for bias in (value, value.expand(1, rows)):
        got = oops.triangle_multiplication(pair, **weights, **{name: bias})
        assert float((got - want).abs().max()) <= TOL[torch.float32] * max(1.0, float(want.abs().max()))
    with pytest.raises(RuntimeError):
        oops.triangle_multiplication(pair, **weights, **{name: value.expand(rows + 1)})


def test_lazily_negated_operands(cuda):
    gen = torch.Generator().manual_seed(9)
    pair, mask = torch.randn(1, 12, 12, 16, generator=gen).to(cuda), torch.rand(1, 12, 12, generator=gen).to(cuda)
    weights = {k: w.to(cuda) for k, w in _weights(gen, 16, 24, True).items()}
    want = oops.triangle_multiplication(-pair, -mask, **{k: -w for k, w in weights.items()})
    got = oops.triangle_multiplication(torch._neg_view(pair), torch._neg_view(mask), **{k: torch._neg_view(w) for k, w in weights.items()})
    assert torch.equal(got, want)
