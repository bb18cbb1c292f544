"""Triangle multiplicative update of pair features, composed from this library's layer norm and library GEMMs.

Mirrors the call surface of the reference's ``triangle_multiplication``
(``oops/pair/triangle_multiplication/triangle_multiplication.py:45-141``) for dense pairs ``(*prefix, N, N, C)``:

    x      = layer_norm(pair)                                        (this library's kernels)
    left   = mask * sigmoid(x Wlg^T + blg) * (x Wlv^T + blv)         right likewise
    update = sum_k left[i, k] * right[j, k]   ("outgoing")   or   sum_k left[k, i] * right[k, j]   ("incoming")
    out    = (layer_norm(update) Wo^T + bo) * sigmoid(x Wog^T + bog)

The five projections of ``x`` are one library GEMM on the stacked weights; the contraction is one batched library GEMM over
channel planes; everything between the GEMMs -- layer norms, gates, mask, the moves between token-major rows and channel
planes -- runs on this library's kernels (``oops_ta_layer_norm_*``, ``oops_ta_pair_gate_*``, ``oops_ta_channel_norm_*``,
``oops_ta_output_gate_*``), each of which reads and writes its operands once, and the reverse pass is written out the same
way.  Calls outside what those kernels serve (see ``_fused_serves``) are composed from single operations.  No kernel of the
contraction itself is built here.  Ragged (NestedTensor) pairs raise ``OOpsUnsupportedError``.
"""

from __future__ import annotations

from typing import Optional

import torch
from torch import Tensor
from torch.nn import functional as F

from ..normalization.layer_norm import check_admission, layer_norm
from ..runtime import proxy_tracing, require_no_forward_mode, require_same_device, tracing, unsupported
from ..runtime.native import native
from ..runtime.nested_tensor import is_nested

_NAME = "triangle_multiplication"


def triangle_multiplication(pair, pair_mask: Optional[Tensor] = None, *, direction: str = "outgoing",
                            input_norm_weight: Tensor, input_norm_bias: Tensor, left_value_weight: Tensor,
                            left_gate_weight: Tensor, right_value_weight: Tensor, right_gate_weight: Tensor,
                            output_norm_weight: Tensor, output_norm_bias: Tensor, output_weight: Tensor,
                            output_gate_weight: Tensor, left_value_bias: Optional[Tensor] = None,
                            left_gate_bias: Optional[Tensor] = None, right_value_bias: Optional[Tensor] = None,
                            right_gate_bias: Optional[Tensor] = None, output_bias: Optional[Tensor] = None,
                            output_gate_bias: Optional[Tensor] = None, input_norm_eps: float = 1e-5,
                            output_norm_eps: float = 1e-5):
    """Incoming or outgoing triangle multiplicative update; see the module docstring."""
    if direction not in ("incoming", "outgoing"):
        raise ValueError(f"{_NAME} direction must be 'incoming' or 'outgoing', got {direction!r}")
    if is_nested(pair) or is_nested(pair_mask):
        raise unsupported(_NAME, "serves dense pairs only (NestedTensor pairs are not built)")
    tensors = (pair, pair_mask, input_norm_weight, input_norm_bias, left_value_weight, left_gate_weight, right_value_weight,
               right_gate_weight, output_norm_weight, output_norm_bias, output_weight, output_gate_weight, left_value_bias,
               left_gate_bias, right_value_bias, right_gate_bias, output_bias, output_gate_bias)
    require_no_forward_mode(_NAME, *tensors)
    require_same_device(_NAME, *tensors)
    if pair.dim() < 3 or pair.shape[-2] != pair.shape[-3]:
        raise ValueError(f"{_NAME} pair must have shape (*prefix, N, N, C) with a square token grid")
    channels = pair.shape[-1]
    hidden = left_value_weight.shape[0]
    expected = {"left_value_weight": (left_value_weight, (hidden, channels)), "left_gate_weight": (left_gate_weight, (hidden, channels)),
                "right_value_weight": (right_value_weight, (hidden, channels)), "right_gate_weight": (right_gate_weight, (hidden, channels)),
                "output_weight": (output_weight, (channels, hidden)), "output_gate_weight": (output_gate_weight, (channels, channels)),
                "input_norm_weight": (input_norm_weight, (channels,)), "input_norm_bias": (input_norm_bias, (channels,)),
                "output_norm_weight": (output_norm_weight, (hidden,)), "output_norm_bias": (output_norm_bias, (hidden,))}
    for name, (tensor, shape) in expected.items():
        if tuple(tensor.shape) != shape:
            raise ValueError(f"{_NAME} {name} must have shape {shape}, got {tuple(tensor.shape)}")
    if not pair.is_cuda:
        raise unsupported(_NAME, "requires CUDA pairs", device=pair.device)

    projections = (left_gate_weight, left_value_weight, right_gate_weight, right_value_weight, output_gate_weight, output_weight)
    biases = (left_gate_bias, left_value_bias, right_gate_bias, right_value_bias, output_gate_bias, output_bias)
    if _fused_serves(pair, pair_mask, hidden, projections, biases):
        for width, weight, bias in ((channels, input_norm_weight, input_norm_bias), (hidden, output_norm_weight, output_norm_bias)):
            if weight.dtype is not bias.dtype or weight.dtype not in (pair.dtype, torch.float32):
                check_admission(pair.new_empty(width), width, weight, bias)  # raises
        norms = [input_norm_weight, input_norm_bias, output_norm_weight, output_norm_bias]
        given = [i for i, bias in enumerate(biases) if bias is not None]
        return native().pair_update(pair, pair_mask, direction == "outgoing", float(input_norm_eps), float(output_norm_eps),
                                    [*norms, *projections, *(biases[i] for i in given)], given)

    x = layer_norm(pair, channels, input_norm_weight, input_norm_bias, input_norm_eps)
    weight = 1.0 if pair_mask is None else pair_mask.to(x.dtype).unsqueeze(-1)
    left = weight * torch.sigmoid(F.linear(x, left_gate_weight.to(x.dtype), _cast(left_gate_bias, x))) * \
        F.linear(x, left_value_weight.to(x.dtype), _cast(left_value_bias, x))
    right = weight * torch.sigmoid(F.linear(x, right_gate_weight.to(x.dtype), _cast(right_gate_bias, x))) * \
        F.linear(x, right_value_weight.to(x.dtype), _cast(right_value_bias, x))
    # channel-major (..., H, N, N) operands of one batched GEMM per prefix element
    if direction == "outgoing":
        a, b = left.movedim(-1, -3), right.movedim(-1, -3).transpose(-1, -2)   # a[h, i, k], b[h, k, j] = right[j, k, h]
    else:
        a, b = left.movedim(-1, -3).transpose(-1, -2), right.movedim(-1, -3)   # a[h, i, k] = left[k, i, h], b[h, k, j]
    update = torch.matmul(a, b).movedim(-3, -1)
    update = layer_norm(update.contiguous(), hidden, output_norm_weight, output_norm_bias, output_norm_eps)
    out = F.linear(update, output_weight.to(x.dtype), _cast(output_bias, x))
    return out * torch.sigmoid(F.linear(x, output_gate_weight.to(x.dtype), _cast(output_gate_bias, x)))


def _cast(bias: Optional[Tensor], like: Tensor) -> Optional[Tensor]:
    return None if bias is None else bias.to(like.dtype)


# ----------------------------------------------------------------------------------------------
# fused passes around the GEMMs
# ----------------------------------------------------------------------------------------------

_DTYPES = (torch.float32, torch.float16, torch.bfloat16)
_PLAIN = (Tensor, torch.nn.Parameter)
_MAX_HIDDEN = 512  # a tile of the channel-norm kernel holds all channels of its tokens in shared memory


def _fused_serves(pair: Tensor, mask: Optional[Tensor], hidden: int, projections, biases) -> bool:
    """Plain eager calls with floating-point parameters, one bias value per projection row (what broadcasts otherwise is
    composed); a mask that takes no gradient and expands to the pair's cells."""
    return (
        pair.dtype in _DTYPES and pair.numel() > 0 and 0 < hidden <= _MAX_HIDDEN and _fits_a_launch(pair) and not _mostly_padding(pair, hidden)
        and type(pair) in _PLAIN and all(type(p) in _PLAIN for p in (*projections, *biases) if p is not None)
        and not torch.compiler.is_compiling() and not torch.is_autocast_enabled("cuda")
        and torch._C._functorch.peek_interpreter_stack() is None and not tracing() and not proxy_tracing()
        and all(p.is_floating_point() for p in projections)
        and all(b is None or (b.is_floating_point() and b.shape == p.shape[:1]) for p, b in zip(projections, biases))
        and (mask is None or (not mask.requires_grad and not mask.is_complex() and mask.dim() < pair.dim()
                              and all(own in (1, want) for own, want in zip(reversed(mask.shape), reversed(pair.shape[:-1])))))
    )


def _fits_a_launch(pair: Tensor) -> bool:
    """Prefix elements are the second grid axis of the passes; cells of a padded plane are counted in 32 bits."""
    tokens, channels = pair.shape[-2:]
    return pair.numel() // (tokens * tokens * channels) <= 65535 and (-(-tokens // 8) * 8) ** 2 < 2**31


def _mostly_padding(pair: Tensor, hidden: int) -> bool:
    """Many small grids, which the passes pad to 8 x 8.

    Up to 2^22 padded cells and channels a call is bound by launches, of which the passes have a third; from 2^23 on they move
    the padding through memory, and the composed form is faster (256 to 4096 grids, 32 to 128 channels, inference / training:
    2 x 2 bf16 1.9 to 3.1 / 1.2 to 2.2 times, 6 x 6 bf16 1.8 / 1.3, 4 x 4 f32 1.1 to 1.2 / 0.9 to 1.2).  Not in 16 bits where
    the tokens are odd in number, so that the composed contraction loads single elements (3 x 3 bf16: 0.38), nor in f32 from
    five tokens on (0.9 and below).
    """
    tokens, channels = pair.shape[-2:]
    if tokens >= 8 or pair.numel() // (tokens * tokens * channels) * 64 * hidden < 2**23:
        return False
    return tokens <= 4 if pair.dtype is torch.float32 else tokens == 1 or tokens % 2 == 0
