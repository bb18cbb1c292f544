"""The tcgen05 kernels for head sizes other than 32 where a row's reference moves or is missing: logits that rise by more than the slack (8) at the
second, third and a later step for some queries of a warp, rows whose first step, or every key, has a bias of -inf, biases of the type's
lowest value; head sizes of one channel group at the lengths at which they are served.  Against f64, with the bounds of
test_wide_kernels_gpu.py; every case asks the library which kernels it takes."""

import pytest
import torch

from oops_b200 import gate_attention_output, pair_bias_attention, triangle_attention
from oops_b200.runtime import cabi
from test_wide_kernels_gpu import close

pytestmark = pytest.mark.gpu


def exact(q, k, v, bias, up):
    """Result and gradients in f64; a row without a finite logit gives zeros."""
    leaves = [t.double().requires_grad_(True) for t in (q, k, v, bias)]
    logits = torch.einsum("brqhd,brkhd->brhqk", leaves[0], leaves[1]) * q.shape[-1] ** -0.5 + leaves[3]
    none = torch.isneginf(logits).all(-1, keepdim=True)
    weights = torch.where(none, 0.0, torch.softmax(torch.where(none, 0.0, logits), -1))
    out = torch.einsum("brhqk,brkhd->brqhd", weights, leaves[2])
    return out, torch.autograd.grad(out, leaves, up.double())


def takes_wide_kernels(q, k, v, bias):
    cols = bias.shape[-1]
    bias = torch.nn.functional.pad(bias.detach(), (0, -cols % 8))[..., :cols]  # (rows of whole words, as the entry point lays them out)
    problem, rows = cabi.make_problem(q, k, v, None, bias, q.shape[-1] ** -0.5), cabi.pair_of(q)
    grads = cabi.Grads(dq=rows, dk=rows, dv=rows, dbias=bias.data_ptr())
    lib = cabi.library()
    return [lib.oops_ta_uses_wide_path(cabi.byref(problem), cabi.byref(rows), g) for g in (None, cabi.byref(grads))]


def check(cuda, q, k, v, bias, up, forward=1, reverse=1):
    leaves = [t.to(cuda).requires_grad_(True) for t in (q, k, v, bias)]
    assert takes_wide_kernels(*leaves) == [forward, reverse]
    out = triangle_attention(*leaves[:3], None, leaves[3])
    grads = torch.autograd.grad(out, leaves, up.to(cuda))
    want, want_grads = exact(q, k, v, bias, up)
    for name, got, ref in zip(("out", "dq", "dk", "dv", "dbias"), (out, *grads), (want, *want_grads)):
        assert bool(torch.isfinite(got).all()), name
        close(name, got, ref)


def operands(rows, cols, heads, dim):
    gen = torch.Generator().manual_seed(cols + dim)
    q, k, v, up = (torch.randn(1, rows, cols, heads, dim, generator=gen).bfloat16() for _ in range(4))
    return q, k, v, torch.randn(1, 1, heads, cols, (cols + 7) // 8 * 8, generator=gen)[..., :cols], up


@pytest.mark.parametrize("rows,cols,heads,dim", [(2, 200, 2, 64), (3, 257, 1, 24), (2, 449, 2, 48), (2, 392, 2, 16)])
def test_rising_logits(cuda, rows, cols, heads, dim):
    q, k, v, bias, up = operands(rows, cols, heads, dim)
    bias[..., ::3, 64:128] += 12  # (queries of every warp, others of it not)
    bias[..., 1::5, 128:192] += 30
    bias[..., 2::7, cols - 3 :] += 60
    bias[..., 4::9, 63] += 100
    bias[..., 6::11, 70] -= 200
    check(cuda, q, k, v, bias.bfloat16(), up)


@pytest.mark.parametrize("rows,cols,heads,dim", [(2, 200, 2, 64), (3, 130, 2, 40), (2, 449, 1, 24)])
@pytest.mark.parametrize("low", [-float("inf"), float(torch.finfo(torch.bfloat16).min)])
def test_low_biases(cuda, rows, cols, heads, dim, low):
    q, k, v, bias, up = operands(rows, cols, heads, dim)
    bias[..., ::3, :64] = low                  # a first step of nothing else
    bias[..., 1::5, :128] = low
    bias[..., 2::7, cols // 64 * 64 :] = low   # a last step
    bias[..., :, 5] = low                      # a key that no query takes
    if low == -float("inf"):
        bias[..., 9, :] = low                  # a query that takes no key
    else:
        bias[..., :, 65] = 0                   # (the norm of a row of lowest values alone is lost in them, and its gradients with it)
    check(cuda, q, k, v, bias.bfloat16(), up)


@pytest.mark.parametrize("rows,cols,heads,dim,forward,reverse", [(2, 520, 2, 8, 1, 1), (2, 392, 3, 16, 1, 1), (20, 260, 4, 8, 1, 1), (20, 264, 4, 16, 1, 1),
                                                                 (2, 256, 2, 16, 0, 0), (40, 128, 4, 16, 0, 1), (1, 64, 2, 64, 0, 1)])
def test_one_channel_group(cuda, rows, cols, heads, dim, forward, reverse):
    q, k, v, bias, up = operands(rows, cols, heads, dim)
    check(cuda, q, k, v, (3 * bias).bfloat16(), up, forward, reverse)


def test_captured_and_hooked(cuda):
    """Token attention and its output step in a captured graph, on new values, and with saved tensors that come back from the host: the bits
    of the eager call."""
    gen = torch.Generator(device=cuda).manual_seed(5)
    shapes = ((2, 8, 300, 64), (2, 8, 300, 64), (2, 8, 300, 64), (1, 8, 300, 304), (2, 300, 384), (512, 384), (384, 512))
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        leaves = [torch.randn(s, device=cuda, generator=gen).mul_(0.3).bfloat16().requires_grad_(True) for s in shapes]
        up = torch.randn(2, 300, 384, device=cuda, generator=gen).bfloat16()

    def call():
        q, k, v, bias, single, gate, output = leaves
        out = gate_attention_output(pair_bias_attention(q, k, v, pair_bias=bias[..., :300]), single, gate, output)
        return out, *torch.autograd.grad(out, leaves, up)

    with torch.cuda.stream(stream):
        for _ in range(3):
            call()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            captured = call()
        with torch.no_grad():
            for leaf in leaves:
                leaf.copy_(torch.randn(leaf.shape, device=cuda, generator=gen).mul_(0.3))
        for _ in range(3):
            graph.replay()
        first = [t.detach().clone() for t in captured]
        with torch.autograd.graph.save_on_cpu():
            hooked = call()
        eager = call()
        for name, a, b, c in zip(("out", "dq", "dk", "dv", "dbias", "dsingle", "dgate", "doutput"), first, eager, hooked):
            assert torch.equal(a, b), name
            assert torch.equal(b, c), name
    stream.synchronize()
