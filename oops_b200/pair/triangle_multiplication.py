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

from ..normalization.layer_norm import _rows_of, backward_rows, check_admission, forward_rows, layer_norm
from ..runtime import cabi, require_no_forward_mode, require_same_device, unsupported
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
    if _fused_serves(pair, pair_mask, hidden, (*projections, *biases)):
        check_admission(pair, channels, input_norm_weight, input_norm_bias)
        check_admission(pair.new_empty(1, dtype=pair.dtype).expand(hidden), hidden, output_norm_weight, output_norm_bias)
        return _FusedUpdate.apply(pair, pair_mask, direction == "outgoing", input_norm_weight, input_norm_bias, input_norm_eps,
                                  output_norm_weight, output_norm_bias, output_norm_eps, *projections, *biases)

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
_MAX_HIDDEN = 512  # a tile of the channel-norm kernel holds all channels of its tokens in shared memory


def _fused_serves(pair: Tensor, mask: Optional[Tensor], hidden: int, parameters) -> bool:
    """Plain eager calls with floating-point parameters; a mask that takes no gradient and expands to the pair's cells."""
    return (
        pair.dtype in _DTYPES and pair.numel() > 0 and 0 < hidden <= _MAX_HIDDEN
        and type(pair) in (Tensor, torch.nn.Parameter)
        and not torch.compiler.is_compiling() and not torch.is_autocast_enabled("cuda")
        and torch._C._functorch.peek_interpreter_stack() is None
        and all(p is None or (p.is_floating_point() and p.dim() in (1, 2)) for p in parameters)
        and (mask is None or (not mask.requires_grad and not mask.is_complex() and mask.dim() < pair.dim()
                              and all(own in (1, want) for own, want in zip(reversed(mask.shape), reversed(pair.shape[:-1])))))
    )


def _run(name: str, device: torch.device, *arguments) -> None:
    with torch.cuda.device(device):
        status = getattr(cabi.library(), name)(*arguments, torch.cuda.current_stream(device).cuda_stream)
    if status:
        raise RuntimeError(f"{_NAME} {name} failed: {cabi.status_message(status)}")


def _address(tensor: Optional[Tensor]) -> Optional[int]:
    return None if tensor is None else tensor.data_ptr()


def _contract(outgoing: bool, left: Tensor, right: Tensor) -> Tensor:
    """update[i, j] = sum_k left[i, k] right[j, k] (outgoing) or sum_k left[k, i] right[k, j], plane by plane."""
    return torch.bmm(left, right.transpose(1, 2)) if outgoing else torch.bmm(left.transpose(1, 2), right)


class _FusedUpdate(torch.autograd.Function):
    @staticmethod
    def forward(ctx, pair, mask, outgoing, in_weight, in_bias, in_eps, out_weight, out_bias, out_eps, *parameters):
        weights, biases = parameters[:6], parameters[6:]
        dtype, device, channels = pair.dtype, pair.device, pair.shape[-1]
        hidden, tokens = weights[0].shape[0], pair.shape[-2]
        prefix = pair.numel() // (tokens * tokens * channels)
        padded = -(-tokens // 8) * 8
        cells, code = prefix * tokens * tokens, cabi.DTYPE_CODE[dtype]
        dims = (prefix, tokens, padded, hidden)
        # rows of the projections: left gate | left value | right gate | right value | output gate
        stacked = torch.cat([w.detach() for w in weights[:5]]).to(dtype)
        stacked_bias = None
        if any(b is not None for b in biases[:5]):
            stacked_bias = torch.cat([w.new_zeros(w.shape[0]) if b is None else b.detach().to(w.dtype)
                                      for w, b in zip(weights[:5], biases[:5])]).to(dtype)
        out_matrix = weights[5].detach().to(dtype)
        rows_in = _rows_of(pair.detach(), channels)
        x, mean1, rstd1 = forward_rows(rows_in, in_weight.detach().contiguous(), in_bias.detach().contiguous(), in_eps)
        proj = F.linear(x, stacked, stacked_bias)
        ld = proj.shape[1]
        weight = None if mask is None else mask.detach().to(dtype).expand(pair.shape[:-1]).contiguous()
        planes = torch.empty((2, prefix * hidden, padded, padded), dtype=dtype, device=device)
        left, right = planes[0], planes[1]
        _run("oops_ta_pair_gate_forward", device, code, *dims, proj.data_ptr(), ld, _address(weight), left.data_ptr(), right.data_ptr())
        update = _contract(outgoing, left, right)
        normed = torch.empty((cells, hidden), dtype=dtype, device=device)
        stats2 = torch.empty((2, cells), dtype=torch.float32, device=device)
        out_w = out_weight.detach().contiguous()
        _run("oops_ta_channel_norm_forward", device, code, cabi.DTYPE_CODE[out_w.dtype], *dims, update.data_ptr(), out_w.data_ptr(),
             out_bias.detach().contiguous().data_ptr(), float(out_eps), normed.data_ptr(), stats2.data_ptr(), stats2[1].data_ptr())
        values = F.linear(normed, out_matrix, None if biases[5] is None else biases[5].detach().to(dtype))
        out = torch.empty(pair.shape, dtype=dtype, device=device)
        gate_at = proj.data_ptr() + 4 * hidden * proj.element_size()
        _run("oops_ta_output_gate_forward", device, code, cells, channels, values.data_ptr(), gate_at, ld, out.data_ptr())
        ctx.set_materialize_grads(False)
        ctx.save_for_backward(rows_in, in_weight.detach().contiguous(), mean1, rstd1, x, stacked, proj, weight, left, right, update, out_w,
                              stats2, normed, out_matrix, values)
        ctx.outgoing, ctx.dims, ctx.shape = outgoing, dims, pair.shape
        ctx.like = [None if p is None else p.dtype for p in parameters]
        return out

    @staticmethod
    def backward(ctx, grad_out):
        if grad_out is None:
            return (None,) * 21
        (rows_in, in_w, mean1, rstd1, x, stacked, proj, weight, left, right, update, out_w, stats2, normed, out_matrix,
         values) = (t if t is None else t.contiguous() for t in ctx.saved_tensors)
        need = ctx.needs_input_grad
        dims, device, code = ctx.dims, proj.device, cabi.DTYPE_CODE[proj.dtype]
        hidden, (cells, ld), channels = dims[3], proj.shape, x.shape[1]
        grads: list = [None] * 21
        dout = _rows_of(grad_out.resolve_neg().to(proj.dtype), channels).contiguous()

        dvalues, dproj = torch.empty_like(values), torch.empty_like(proj)
        gate_offset = 4 * hidden * proj.element_size()
        _run("oops_ta_output_gate_backward", device, code, cells, channels, dout.data_ptr(), values.data_ptr(),
             proj.data_ptr() + gate_offset, ld, dvalues.data_ptr(), dproj.data_ptr() + gate_offset, ld)
        if need[14]:
            grads[14] = (dvalues.t() @ normed).to(ctx.like[5])
        if need[20]:
            grads[20] = dvalues.sum(0).to(ctx.like[11])
        dnormed = dvalues @ out_matrix
        dupdate = torch.empty_like(update)
        dw2 = torch.empty_like(out_w) if need[6] else None
        db2 = torch.empty_like(out_w) if need[7] else None
        nbytes = cabi.library().oops_ta_channel_norm_backward_workspace_bytes(code, *dims)
        scratch = torch.empty(int(nbytes), dtype=torch.uint8, device=device)
        _run("oops_ta_channel_norm_backward", device, code, cabi.DTYPE_CODE[out_w.dtype], *dims, dnormed.data_ptr(), update.data_ptr(),
             out_w.data_ptr(), stats2.data_ptr(), stats2[1].data_ptr(), dupdate.data_ptr(), _address(dw2), _address(db2),
             scratch.data_ptr(), int(nbytes))
        grads[6], grads[7] = dw2, db2
        if not any(need[i] for i in (0, 3, 4, *range(9, 14), *range(15, 20))):
            return tuple(grads)
        if ctx.outgoing:
            dleft, dright = torch.bmm(dupdate, right), torch.bmm(dupdate.transpose(1, 2), left)
        else:
            dleft, dright = torch.bmm(right, dupdate.transpose(1, 2)), torch.bmm(left, dupdate)
        _run("oops_ta_pair_gate_backward", device, code, *dims, proj.data_ptr(), ld, _address(weight), dleft.data_ptr(),
             dright.data_ptr(), dproj.data_ptr(), ld)
        extents = [hidden] * 4 + [channels]
        if any(need[9:14]):
            stacked_grad = dproj.t() @ x
            for i, piece in enumerate(stacked_grad.split(extents)):
                if need[9 + i]:
                    grads[9 + i] = piece.to(ctx.like[i])
        if any(need[15:20]):
            for i, piece in enumerate(dproj.sum(0).split(extents)):
                if need[15 + i]:
                    grads[15 + i] = piece.to(ctx.like[6 + i])
        if need[0] or need[3] or need[4]:
            dx, grads[3], grads[4] = backward_rows(dproj @ stacked, rows_in, in_w, mean1, rstd1, in_w.dtype, need[0], need[3], need[4])
            grads[0] = None if dx is None else dx.view(ctx.shape)
        return tuple(grads)
