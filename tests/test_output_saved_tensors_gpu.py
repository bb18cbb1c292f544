"""Saved tensors of the output step that come back through hooks as something else: another type, size or device raises (a value of theirs
is never read as if it fitted), another layout of the same values gives the same gradients; batched gradients and dispatch modes
reach the library's products."""

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from oops_b200 import gate_attention_output

pytestmark = pytest.mark.gpu
SAVED = ("attention", "single", "gate_weight", "output_weight", "gate", "gated")  # in the order in which the node saves them


def leaves_and_upstream(device):
    gen = torch.Generator(device=device).manual_seed(3)
    shapes = ((2, 4, 24, 16), (2, 24, 40), (64, 40), (48, 64))
    leaves = [torch.randn(*s, device=device, generator=gen).mul_(0.3).bfloat16().requires_grad_(True) for s in shapes]
    return leaves, torch.randn(2, 24, 48, device=device, generator=gen).bfloat16()


def with_hook(leaves, upstream, which, change):
    count = iter(range(len(SAVED)))

    def pack(t):
        return SAVED[next(count)], t.detach()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda kept: change(kept[1]) if kept[0] == which else kept[1]):
        out = gate_attention_output(*leaves)
    return torch.autograd.grad(out, leaves, upstream)


@pytest.mark.parametrize("which", ("single", "gate", "gated"))
@pytest.mark.parametrize("change", (lambda t: t.float(), lambda t: t.half(), lambda t: t.cpu(), lambda t: t[..., :-8].contiguous(),
                                    lambda t: t[:1].contiguous()), ids=("f32", "f16", "cpu", "narrow", "short"))
def test_what_does_not_fit_raises(cuda, which, change):
    leaves, upstream = leaves_and_upstream(cuda)
    with pytest.raises(RuntimeError):
        with_hook(leaves, upstream, which, change)


@pytest.mark.parametrize("which", SAVED)
def test_other_layouts_of_the_same_values(cuda, which):
    leaves, upstream = leaves_and_upstream(cuda)
    want = with_hook(leaves, upstream, which, lambda t: t)

    def strided(t):
        return t.transpose(-1, -2).contiguous().transpose(-1, -2)

    def off_a_word(t):
        return torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)

    for change in (strided, off_a_word):
        for got, ref in zip(with_hook(leaves, upstream, which, change), want):  # (sums in another order)
            assert float((got.double() - ref.double()).norm()) <= 2.0**-7 * float(ref.double().norm())


def test_batched_gradients(cuda):
    """The gradient of the weight behind the gate is a plain product, which takes a batch of upstream gradients."""
    leaves, upstream = leaves_and_upstream(cuda)
    batch = torch.stack([upstream, -2 * upstream])
    got, = torch.autograd.grad(gate_attention_output(*leaves), [leaves[3]], batch, is_grads_batched=True)
    for one, up in zip(got, batch):
        want, = torch.autograd.grad(gate_attention_output(*leaves), [leaves[3]], up)
        assert float((one.double() - want.double()).norm()) <= 2.0**-7 * float(want.double().norm())


def test_a_dispatch_mode_sees_the_products_of_the_reverse(cuda):
    leaves, upstream = leaves_and_upstream(cuda)
    seen = []

    class Recorder(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    out = gate_attention_output(*leaves)
    with Recorder():
        torch.autograd.grad(out, leaves, upstream)
    assert torch.ops.aten.mm.default in seen
