"""Calls that something records: ``torch.jit.trace`` and ``make_fx`` must take the operator itself into their graph, not the
memory that its launch filled while they looked on, or refuse; a dispatch mode that only looks on changes nothing."""

import pytest
import torch
from torch.fx.experimental.proxy_tensor import make_fx
from torch.utils._python_dispatch import TorchDispatchMode

import oops_b200 as oops

pytestmark = pytest.mark.gpu


def operands(name, device, scale):
    gen = torch.Generator().manual_seed(len(name))

    def draw(*shape):
        return (scale * torch.randn(*shape, generator=gen)).to(device, torch.bfloat16)

    mask = (torch.rand(1, 5, 24, generator=gen) > 0.3).to(device)
    pair = [draw(1, 5, 24, 2, 32) for _ in range(4)]
    return {
        "attention": (pair[:3], lambda q, k, v: oops.triangle_attention(q, k, v, mask)),
        "gated": (pair, lambda q, k, v, g: oops.triangle_attention_gated(q, k, v, g, mask)),
        "norm": ([draw(6, 32), draw(32), draw(32)], lambda x, w, b: oops.layer_norm(x, 32, w, b)),
        "plain norm": ([draw(6, 32)], lambda x: oops.layer_norm(x, 32)),
        "gate": ([draw(2, 2, 8, 16), draw(2, 8, 24), draw(32, 24), draw(24, 32)], oops.gate_attention_output),
    }[name]


OPERATORS = ["attention", "gated", "norm", "plain norm", "gate"]


def with_grads(f, values):
    leaves = [v.detach().requires_grad_(True) for v in values]
    out = f(*leaves)
    return [out.detach(), *torch.autograd.grad(out, leaves, torch.ones_like(out))]


def same(got, want):
    for a, b in zip(got, want):  # the same kernels on the same values; "gated" rounds once more on its way through the trace
        assert float((a.float() - b.float()).norm()) <= 2.0**-8 * float(b.float().norm())


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("name", OPERATORS)
def test_a_traced_call_follows_its_inputs(cuda, name):
    first, f = operands(name, cuda, 1.0)
    second, _ = operands(name, cuda, 0.5)
    traced = torch.jit.trace(f, tuple(v.requires_grad_(True) for v in first), check_trace=False)
    same(with_grads(traced, second), with_grads(f, second))
    with torch.no_grad():
        same([traced(*second)], [f(*second)])


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("name", OPERATORS)
def test_make_fx_records_the_operator_or_refuses(cuda, name):
    first, f = operands(name, cuda, 1.0)
    second, _ = operands(name, cuda, 0.5)
    if name == "attention":
        same([make_fx(f)(*first)(*second)], [f(*second)])
    else:
        with pytest.raises(oops.OOpsUnsupportedError):
            make_fx(f)(*first)


@pytest.mark.parametrize("name", OPERATORS)
def test_a_dispatch_mode_may_look_on(cuda, name):
    class Looker(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    values, f = operands(name, cuda, 1.0)
    want = with_grads(f, values)
    with Looker():
        got = with_grads(f, values)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
