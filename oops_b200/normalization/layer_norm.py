"""Layer normalisation over the final feature axis, with the reference's call surface.

Mirrors ``oops/normalization/layer_norm/layer_norm.py:37-154`` of the reference: CUDA float16 / bfloat16 / float32
activations ``(..., C)`` with ``1 <= C <= 8192`` (or a packed ragged batch whose last element axis is static and
physically last), optional ``weight`` / ``bias`` of shape ``(C,)`` in the activation dtype or, for 16-bit activations,
float32.  The kernels are ``oops_ta_layer_norm_forward/_backward`` of the C ABI (``include/oops_ta.h``); there is no
fallback.  Differences from the reference: activations are viewed as ``(rows, C)`` with contiguous rows (other
layouts are copied once, as ``Tensor.reshape`` does); autocast promotion is not re-implemented (parameters must already
be of an accepted dtype); the call is not registered as a ``torch.compile`` custom op.
"""

from __future__ import annotations

import math
from typing import Iterable, Optional

import torch
from torch import Tensor
from torch.autograd import forward_ad

from ..runtime import require_no_forward_mode, require_no_proxy_tracing, require_same_device, tracing, unsupported
from ..runtime.native import native
from ..runtime.nested_tensor import is_nested

_NAME = "layer_norm"
_MAX_WIDTH = 8192
_DTYPE_CODES = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}
_HALF = (torch.float16, torch.bfloat16)


def layer_norm(input, normalized_shape, weight: Optional[Tensor] = None, bias: Optional[Tensor] = None, eps: float = 1e-5):
    """Normalize the final feature dimension of CUDA activations; see the module docstring."""
    width = normalized_shape if isinstance(normalized_shape, int) else None
    if width is not None and forward_ad._current_level < 0:
        out = native().layer_norm(input, width, weight, bias, eps)
        if out is not None:
            return out
    if is_nested(input):
        return _layer_norm_nested(input, normalized_shape, weight, bias, eps)
    require_no_forward_mode(_NAME, input, weight, bias)
    require_same_device(_NAME, input, weight, bias)
    check_admission(input, normalized_shape, weight, bias)
    input, weight, bias = (t if t is None else t.resolve_neg() for t in (input, weight, bias))
    require_no_proxy_tracing(_NAME)
    eps = float(eps)
    if tracing():
        return _TracedLayerNorm.apply(input, weight, bias, eps)
    out = None
    if torch._C._functorch.peek_interpreter_stack() is None:
        out = native().layer_norm_node(input, input.shape[-1], weight, bias, eps)
    if out is None:  # served layouts behind a transform or a tensor subclass
        raise unsupported(_NAME, "does not support torch.func transforms or dispatching tensor subclasses")
    return out


class _TracedLayerNorm(torch.autograd.Function):
    """The node as ``torch.jit.trace`` can record it."""

    @staticmethod
    def forward(ctx, x, weight, bias, eps):
        out, stats = native().layer_norm_forward(x, weight, bias, eps)
        ctx.save_for_backward(x, weight, bias, stats)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        x, weight, bias, stats = ctx.saved_tensors
        need = [ctx.needs_input_grad[0], weight is not None and ctx.needs_input_grad[1], bias is not None and ctx.needs_input_grad[2]]
        return (*native().layer_norm_backward(grad_out, x, weight, bias, stats, need), None)


def check_admission(input, normalized_shape, weight: Optional[Tensor], bias: Optional[Tensor]) -> None:
    """Raise ``OOpsUnsupportedError`` for what the kernels do not serve."""
    shape = (normalized_shape,) if isinstance(normalized_shape, int) else tuple(normalized_shape)
    if len(shape) != 1:
        raise unsupported(_NAME, "normalizes over the final dimension only", normalized_shape=shape, input_shape=tuple(input.shape))
    width = math.prod(shape)
    affine = [p for p in (weight, bias) if p is not None]
    mixed = input.dtype in _HALF and any(p.dtype is torch.float32 for p in affine) and any(p.dtype is not torch.float32 for p in affine)
    supported = (
        input.is_cuda and input.dim() >= 1 and input.shape[-1] == width and 0 < width <= _MAX_WIDTH and input.dtype in _DTYPE_CODES
        and not mixed
        and all(p.shape == (width,) and (p.dtype is input.dtype or (input.dtype in _HALF and p.dtype is torch.float32)) for p in affine)
    )
    if not supported:
        raise unsupported(_NAME, "requires a CUDA half/float32 activation with a matching contiguous affine row",
                          input_dtype=input.dtype, device=input.device, normalized_size=width,
                          weight_dtype=None if weight is None else weight.dtype, bias_dtype=None if bias is None else bias.dtype)
    if input.numel() == 0:
        raise unsupported(_NAME, "does not serve an empty input", input_shape=tuple(input.shape))


def _layer_norm_nested(input, normalized_shape, weight, bias, eps):
    if is_nested(weight) or is_nested(bias):
        raise ValueError(f"{_NAME} NestedTensor input requires dense affine parameters")
    if input.dim() < 2 or not input.ragged_dims:
        raise unsupported(_NAME, "requires a NestedTensor with explicit packed element topology", ragged_dims=input.ragged_dims)
    normalized_dim = input.dim() - 2
    if normalized_dim in input.ragged_dims or input.packed_dim_order[-1] != normalized_dim:
        raise unsupported(_NAME, "requires the final logical element dimension to be static and physically last",
                          ragged_dims=input.ragged_dims, packed_dim_order=input.packed_dim_order)
    packed = input.concat
    if packed.dim() < 1:
        raise unsupported(_NAME, "requires packed values with a retained static final dimension")
    shape: Iterable[int] = (normalized_shape,) if isinstance(normalized_shape, int) else tuple(normalized_shape)
    return input.packed_like(layer_norm(packed, shape, weight, bias, eps))
