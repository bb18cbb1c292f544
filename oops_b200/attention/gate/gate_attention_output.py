"""``gate_attention_output`` and the gate fused into triangle attention's epilogue.

``gate_attention_output`` keeps the signature, argument meaning and error texts of
``oops/attention/gate/gate_attention_output.py:36-100`` (shape contract ``_contract.py:27-48``,
math ``composed.py:47-53``): ``linear(sigmoid(linear(single, gate_weight)) * attention_flat, output_weight)``.
The two linear maps are plain library GEMMs; the element-wise core between them -- the sigmoid gate on the
attention values, including the move from the head-major ``(*, H, Q, D)`` attention layout to the token-major
``(*, Q, H*D)`` layout of the projection -- is a hand-written kernel behind the C ABI
(``oops_ta_gate_forward`` / ``oops_ta_gate_backward``).

``triangle_attention_gated`` is the fused form this library adds: triangle attention whose forward kernel applies
the gate to its output tile while it is still in registers, so the ``(*, R, C, H*D)`` attention values are never
written and re-read between the two operators at inference, and only written once more (for the reverse pass) in
training.  Dense inputs only; ragged (NestedTensor) operands of the reference's gate operator are not served.
"""

from __future__ import annotations

from typing import Optional

import torch
from torch import Tensor
from torch.autograd import forward_ad
from torch.nn import functional as F

from ...runtime import cabi, require_no_forward_mode, require_no_proxy_tracing, require_same_device, result_like, tracing, unsupported
from ...runtime.native import native
from ...runtime.nested_tensor import is_nested
from ..triangle import function as _function
from ..triangle.triangle_attention import (
    _check_admission, _check_dense_shapes, _flags, _require_bool_mask, _unit_inner,
)

_OPERATOR = "gate_attention_output"


def _check_gate_output(attention: Tensor, single: Tensor, gate_weight: Tensor, output_weight: Tensor) -> None:
    """Shape contract of the reference (oops/attention/gate/_contract.py:27-48), same messages."""
    rank = attention.dim()
    if rank not in (3, 4, 5):
        raise ValueError(
            "attention must have layout (num_heads, query_length, head_size) under optional batch and sample axes"
        )
    if single.dim() + 1 != rank:
        raise ValueError("single must have layout (..., query_length, single_channels)")
    if gate_weight.dim() != 2 or output_weight.dim() != 2:
        raise ValueError("gate_weight and output_weight must be rank-2 matrices")
    lead, (heads, length, head_size) = tuple(attention.shape[:-3]), tuple(attention.shape[-3:])
    channels = heads * head_size
    if tuple(single.shape[:-1]) != (*lead, length):
        raise ValueError("single must share the attention leading axes and its query_length")
    if tuple(gate_weight.shape) != (channels, single.shape[-1]):
        raise ValueError("gate_weight must have shape (num_heads * head_size, single_channels)")
    if output_weight.shape[1] != channels:
        raise ValueError("output_weight input channels must equal num_heads * head_size")


def _run_gate(attention5: Tensor, gate5: Tensor, out5: Tensor) -> None:
    """``out5 = sigmoid(gate5) * attention5`` on ``(B, R, C, H, D)`` views."""
    native().run_gate(attention5, gate5, out5)


class _TracedGate(torch.autograd.Function):
    """``sigmoid(gate5) * attention5`` on ``(B, R, C, H, D)`` values, as ``torch.jit.trace`` can record it."""

    @staticmethod
    def forward(ctx, attention5, gate5):
        attention5, gate5 = _unit_inner(attention5), _unit_inner(gate5)
        out5 = torch.empty(gate5.shape, dtype=gate5.dtype, device=gate5.device)
        _run_gate(attention5, gate5, out5)
        ctx.save_for_backward(attention5, gate5)
        return out5

    @staticmethod
    def backward(ctx, grad5):
        attention5, gate5 = (_unit_inner(t) for t in ctx.saved_tensors)
        d_attention, d_gate = (torch.empty(t.shape, dtype=t.dtype, device=t.device) for t in (attention5, gate5))
        native().run_gate_backward(attention5, gate5, _unit_inner(grad5.resolve_neg().to(gate5.dtype)), d_attention, d_gate)
        return d_attention, d_gate


def _sigmoid_gate(attention4: Tensor, gate: Tensor) -> Tensor:
    """``sigmoid(gate) * attention`` for ``(B, H, Q, D)`` attention and ``(B, Q, H * D)`` gate."""
    if not tracing():
        return result_like(native().sigmoid_gate(attention4, gate), gate)
    heads, head_size = int(attention4.shape[1]), int(attention4.shape[3])
    gated5 = _TracedGate.apply(attention4.permute(0, 2, 1, 3).unsqueeze(1), gate.unflatten(-1, (heads, head_size)).unsqueeze(1))
    return gated5.squeeze(1).flatten(-2)


def gate_attention_output(attention, single, gate_weight: Tensor, output_weight: Tensor):
    r"""Apply a sigmoid gate and output projection to head-major attention values.

    ``linear(sigmoid(linear(single, gate_weight)) * attention_flat, output_weight)`` where ``attention_flat`` puts the
    heads and channels of a query token next to each other.

    Args:
        attention: dense ``(*prefix, H, Q, D)`` values of rank 3, 4 or 5.
        single: gating input ``(*prefix, Q, C)`` on the attention device.
        gate_weight: ``(H * D, C)``; output_weight: ``(O, H * D)``.

    Returns:
        ``(*prefix, Q, O)``.

    Raises:
        ValueError: ranks, shapes, devices or dense/ragged representations disagree.
        OOpsUnsupportedError: ragged operands, non-CUDA tensors, unsupported dtypes.
    """
    if not torch.compiler.is_compiling() and forward_ad._current_level < 0:
        out = native().gate_attention_output(attention, single, gate_weight, output_weight)
        if out is not None:
            return out
    if is_nested(attention) or is_nested(single):
        if is_nested(attention) != is_nested(single):
            raise ValueError(
                "gate_attention_output nested attention requires a NestedTensor single"
                if is_nested(attention) else "gate_attention_output dense attention cannot use a NestedTensor single"
            )
        raise unsupported(_OPERATOR, "does not serve NestedTensor operands in this library (dense inputs only)")
    _check_gate_output(attention, single, gate_weight, output_weight)
    require_same_device(_OPERATOR, attention, single, gate_weight, output_weight)
    require_no_forward_mode(_OPERATOR, attention, single, gate_weight, output_weight)
    if not attention.is_cuda or attention.dtype not in cabi.DTYPE_CODE or single.dtype != attention.dtype:
        raise unsupported(
            _OPERATOR, "requires CUDA float16/bfloat16/float32 attention and single of one dtype",
            attention=f"{tuple(attention.shape)} {attention.dtype} {attention.device}", single_dtype=single.dtype,
        )
    require_no_proxy_tracing(_OPERATOR)
    lead = tuple(attention.shape[:-3])
    attention4 = attention.reshape(-1, *attention.shape[-3:]) if len(lead) != 1 else attention
    single3 = single.reshape(-1, *single.shape[-2:]) if len(lead) != 1 else single
    gate = F.linear(single3, gate_weight.to(single3.dtype)).to(attention.dtype)  # (autocast has a type of its own)
    gated = _sigmoid_gate(attention4, gate)
    result = F.linear(gated, output_weight.to(gated.dtype))
    return result.reshape(*lead, *result.shape[-2:]) if len(lead) != 1 else result


# ----------------------------------------------------------------------------------------------
# the gate fused into triangle attention
# ----------------------------------------------------------------------------------------------


def triangle_attention_gated(query: Tensor, key: Tensor, value: Tensor, gate: Tensor, mask: Optional[Tensor] = None,
                             triangle_bias: Optional[Tensor] = None, *, scale: Optional[float] = None) -> Tensor:
    r"""``sigmoid(gate) * triangle_attention(query, key, value, mask, triangle_bias, scale=scale)`` in one forward kernel.

    ``gate`` holds the gate logits of the output projection, ``linear(pair, gate_weight)``, with the query's shape
    ``(B, R, C, H, D)`` (or ``(B, R, C, H * D)``); the result has the query's shape and feeds the output projection.
    Dense rank-5 inputs; everything else as ``triangle_attention``.  Gradients flow to query, key, value, gate and bias.
    """
    operator = "triangle_attention_gated"
    if not torch.compiler.is_compiling() and forward_ad._current_level < 0:
        out = native().triangle_attention_gated(query, key, value, gate, mask, triangle_bias, scale, _flags())
        if out is not None:
            return out
    for operand in (query, key, value, gate, mask, triangle_bias):
        if operand is not None and is_nested(operand):
            raise unsupported(operator, "serves dense inputs only")
    if query.dim() != 5:
        raise ValueError(f"{operator} query must be (batch, rows, cols, num_heads, head_size), got rank {query.dim()}")
    _check_dense_shapes(query, key, value, mask, triangle_bias)
    if gate.dim() == 4 and gate.shape[-1] == query.shape[-2] * query.shape[-1]:
        gate = gate.unflatten(-1, tuple(query.shape[-2:]))
    if tuple(gate.shape) != tuple(query.shape) or gate.dtype != query.dtype:
        raise ValueError(f"{operator} gate must have the query's shape {tuple(query.shape)} and dtype, got {tuple(gate.shape)} {gate.dtype}")
    require_same_device(operator, query, key, value, gate, mask, triangle_bias)
    require_no_forward_mode(operator, query, key, value, gate, triangle_bias)
    _require_bool_mask(mask)
    _check_admission(query, key, value, mask, triangle_bias,
                     "requires CUDA float16/bfloat16/float32 q/k/v of one dtype and shape with head_size <= 256")
    batch, rows, cols, _heads, head_size = query.shape
    q5 = _function.DenseGeometry().canonical_pair(_unit_inner(query))
    k5 = q5 if key is query else _function.DenseGeometry().canonical_pair(_unit_inner(key))
    v5 = q5 if value is query else k5 if value is key else _function.DenseGeometry().canonical_pair(_unit_inner(value))
    g5 = _unit_inner(gate)
    mask3 = None if mask is None else mask.expand(batch, rows, cols)
    bias5 = None
    if triangle_bias is not None:
        bias5 = triangle_bias.resolve_neg().resolve_conj().contiguous()
        if bias5.element_size() == 2 and cols % 8 != 0:
            bias5 = torch.nn.functional.pad(bias5, (0, -cols % 8))[..., :cols]
    scale = float(head_size**-0.5 if scale is None else scale)
    require_no_proxy_tracing(operator)
    if tracing():
        plain = _function.TracedAttention.apply(q5, k5, v5, mask3, bias5, scale, _function.DenseGeometry(), _flags())
        return _TracedGate.apply(plain, g5)
    return native().gated_attend(q5, k5, v5, g5, mask3, bias5, scale, _flags())


__all__ = ["gate_attention_output", "triangle_attention_gated"]
