"""Autograd boundary of triangle attention over the C ABI.

Takes the place of ``oops/attention/triangle/triton/ops.py`` in the reference
(``_TriangleAttention`` :413, ``_setup_context`` :369, ``_backward_from_context``
:380): gradients for query, key, value and bias only; mask and the saved
log-sum-exp are not differentiable; undefined upstream gradients are not
materialised; the reverse pass honours ``needs_input_grad`` subsets; no double
backward.

The autograd node itself is compiled (``oops_b200/csrc/native.cpp``); this module
describes calls to it and registers the dispatcher route.
A call is described by a *geometry*: a recipe that turns the tensors handed to
the node into one or more uniform ``(B, R, C, H, D)`` views, each of which is
one C-ABI problem.  Dense inputs are a single view (the tensor itself, whatever
its strides).  A packed ragged batch is one view per sample, computed from the
packed layout the reference documents in ``oops/attention/triangle/nested.py:
275-288`` (cell start, cell stride = number of prefixes, bias start/strides).
"""

from __future__ import annotations

from contextlib import contextmanager
from dataclasses import dataclass
from typing import List, Optional, Sequence, Tuple

import torch
from torch import Tensor

from ...runtime import cabi, proxy_tracing, result_like, tracing, unsupported
from ...runtime.native import native


@dataclass(frozen=True)
class DenseGeometry:
    """One uniform problem: the tensors are already ``(B, R, C, H, D)`` views."""

    def canonical_pair(self, tensor: Tensor) -> Tensor:
        """Unit inner stride; 16-bit tensors additionally get 16-byte aligned rows, which the TMA kernels need."""
        if tensor.shape[-1] != 1 and tensor.stride(-1) != 1:
            return tensor.contiguous()
        if tensor.element_size() == 2 and (
            tensor.data_ptr() % 16 != 0
            or any(size > 1 and (stride <= 0 or stride % 8 != 0) for size, stride in zip(tensor.shape[:-1], tensor.stride()[:-1]))
        ):
            return tensor.contiguous()
        return tensor

    def canonical_bias(self, bias: Tensor) -> Tensor:
        return bias


@dataclass(frozen=True)
class NestedGeometry:
    """Packed ragged batch of square samples.

    Pair tensors are ``(cells, P, H, D)`` contiguous, masks ``(cells, P)``, and the
    bias is head-major ``(P, H, bias_values)`` with each sample's block laid out as
    ``(groups, query, key)``.  ``transposed`` means that the packed cell order is
    column-major (the ending-node form).
    """

    lengths: Tuple[int, ...]
    prefixes: int
    transposed: bool
    bias_groups: Tuple[int, ...] = ()
    bias_row_strides: Tuple[int, ...] = ()  # key-axis stride of each sample's bias rows (>= N_i; padded for alignment)

    def _cell_starts(self) -> List[int]:
        starts, at = [], 0
        for n in self.lengths:
            starts.append(at)
            at += n * n
        return starts

    def pair_views(self, tensor: Tensor) -> List[Tensor]:
        """The samples of a packed pair tensor as (P, N_i, N_i, H, D) views, as the compiled host layer addresses them."""
        _, prefixes, heads, dim = tensor.shape
        cell = prefixes * heads * dim
        views = []
        for n, start in zip(self.lengths, self._cell_starts()):
            major, minor = n * cell, cell
            row_stride, col_stride = (minor, major) if self.transposed else (major, minor)
            views.append(
                tensor.as_strided(
                    (prefixes, n, n, heads, dim),
                    (heads * dim, row_stride, col_stride, dim, 1),
                    tensor.storage_offset() + start * cell,
                )
            )
        return views

    def canonical_pair(self, tensor: Tensor) -> Tensor:
        return tensor.contiguous()

    def canonical_bias(self, bias: Tensor) -> Tensor:
        return bias.contiguous()


@contextmanager
def checked_device_status(enabled: bool = True):
    """Inside the block every forward and reverse call ends by synchronising with the device and reading the
    library's device-side status word; a kernel that gave up one of its bounded waits (its outputs are then
    undefined) raises ``RuntimeError`` and the word is cleared.  Off by default because of the synchronisation:
    production callers poll ``oops_b200.runtime.cabi.device_status()`` at a point where they synchronise anyway."""
    previous = native().check_device_status(enabled)
    try:
        yield
    finally:
        native().check_device_status(previous)


def run_forward(
    geometry, query: Tensor, key: Tensor, value: Tensor, mask: Optional[Tensor], bias: Optional[Tensor], scale: float,
    flags: int, want_lse: bool,
) -> Tuple[Tensor, Optional[Tensor]]:
    """Launch the forward pass of every view; returns ``(out, lse)``."""
    return native().run_forward(encode_geometry(geometry), query, key, value, mask, bias, scale, flags, want_lse)


def backward_scratch_bytes(query, key, value, mask, bias, scale, flags, need) -> int:
    """Scratch bytes the reverse pass of one dense ``(B, R, C, H, D)`` problem needs for this gradient request."""
    lib = cabi.library()
    problem = cabi.make_problem(query, key, value, mask, bias, scale, flags)
    grads = cabi.Grads()
    marker = cabi.Pair(1, 0, 0, 0, 0)  # the size query looks at which pointers are set, not at what they point to
    none = cabi.Pair(None, 0, 0, 0, 0)
    grads.dq, grads.dk, grads.dv = (marker if need[0] else none, marker if need[1] else none, marker if need[2] else none)
    if need[3] and bias is not None:
        grads.dbias = 1
    return int(lib.oops_ta_backward_workspace_bytes(cabi.byref(problem), cabi.byref(grads)))


def run_backward(
    geometry, grad_out: Tensor, query: Tensor, key: Tensor, value: Tensor, mask: Optional[Tensor],
    bias: Optional[Tensor], out: Tensor, lse: Tensor, scale: float, flags: int, need: Sequence[bool],
    *, scratch: Optional[Tensor] = None, dbias_dtype: Optional[torch.dtype] = None,
) -> Tuple[Optional[Tensor], Optional[Tensor], Optional[Tensor], Optional[Tensor]]:
    """Launch the reverse pass of every view; returns ``(dq, dk, dv, dbias)``.

    ``scratch`` lends a caller-owned byte buffer to the call (it must be large enough for every view; without it one
    buffer per view is allocated).  ``dbias_dtype`` overrides the type of the bias gradient buffer: ``torch.float32``
    together with ``cabi.FLAG_DBIAS_F32`` in ``flags`` returns the unrounded f32 sums of a row-shared bias."""
    return native().run_backward(
        encode_geometry(geometry), grad_out, query, key, value, mask, bias, out, lse, scale, flags, list(need), scratch,
        dbias_dtype is torch.float32,
    )


# ----------------------------------------------------------------------------------------------
# Dispatcher route: torch.library custom ops with fake (meta) implementations, used under torch.compile and
# FakeTensorMode, where tensors carry no data pointers.  Takes the place of the reference's
# `ooperators::_triangle_attention_forward/_backward` ops and their `register_fake` shape functions
# (oops/attention/triangle/triton/ops.py:156-366).  Eager calls keep the compiled
# autograd node (native.cpp), and torch.jit.trace gets a Python one.
# ----------------------------------------------------------------------------------------------


def encode_geometry(geometry) -> List[int]:
    """Flatten a geometry into integers (custom-op schemas carry no Python objects)."""
    if isinstance(geometry, DenseGeometry):
        return []
    count = len(geometry.lengths)
    groups = geometry.bias_groups or (0,) * count
    rows = geometry.bias_row_strides or geometry.lengths
    return [geometry.prefixes, int(geometry.transposed), count, int(bool(geometry.bias_groups)), *geometry.lengths, *groups,
            *rows]


def decode_geometry(code: Sequence[int]):
    if len(code) == 0:
        return DenseGeometry()
    prefixes, transposed, count, has_bias = (int(v) for v in code[:4])
    lengths = tuple(int(v) for v in code[4 : 4 + count])
    groups = tuple(int(v) for v in code[4 + count : 4 + 2 * count]) if has_bias else ()
    rows = tuple(int(v) for v in code[4 + 2 * count : 4 + 3 * count]) if has_bias else ()
    return NestedGeometry(lengths=lengths, prefixes=prefixes, transposed=bool(transposed), bias_groups=groups,
                          bias_row_strides=rows)


def _reverse_of_saved(geometry, grad_out, query, key, value, mask, bias, out, lse, scale, flags, need):
    """``run_backward`` on what was saved for it, whose strides hooks or a recorded graph may have changed."""
    query, key, value, out = (geometry.canonical_pair(t) for t in (query, key, value, out))
    grad_out = geometry.canonical_pair(grad_out.resolve_neg().to(query.dtype))
    if bias is not None:
        bias = geometry.canonical_bias(bias)
    if mask is not None and not isinstance(geometry, DenseGeometry):
        mask = mask.contiguous()
    return run_backward(geometry, grad_out, query, key, value, mask, bias, out, lse.contiguous(), scale, flags, need)


class TracedAttention(torch.autograd.Function):
    """The node as ``torch.jit.trace`` can record it."""

    @staticmethod
    def forward(ctx, query, key, value, mask, bias, scale, geometry, flags):
        ctx.set_materialize_grads(False)
        wanted = any(ctx.needs_input_grad[i] for i in (0, 1, 2, 4))
        out, lse = run_forward(geometry, query, key, value, mask, bias, scale, flags, want_lse=wanted)
        if wanted:
            ctx.save_for_backward(query, key, value, mask, bias, out, lse)
            ctx.scale, ctx.geometry, ctx.flags = scale, geometry, flags
        return out

    @staticmethod
    def backward(ctx, grad_out):
        if grad_out is None:
            return (None,) * 8
        query, key, value, mask, bias, out, lse = ctx.saved_tensors
        need = tuple(ctx.needs_input_grad[i] for i in (0, 1, 2, 4))
        dq, dk, dv, dbias = _reverse_of_saved(ctx.geometry, grad_out, query, key, value, mask, bias, out, lse, ctx.scale, ctx.flags, need)
        return dq, dk, dv, None, dbias, None, None, None


@torch.library.custom_op("oops_b200::triangle_attention_forward", mutates_args=())
def _forward_op(
    query: Tensor, key: Tensor, value: Tensor, mask: Optional[Tensor], bias: Optional[Tensor], scale: float,
    geometry: List[int], flags: int, want_lse: bool,
) -> Tuple[Tensor, Tensor]:
    out, lse = run_forward(decode_geometry(geometry), query, key, value, mask, bias, scale, flags, want_lse)
    if lse is None:
        lse = torch.empty(0, dtype=torch.float32, device=query.device)
    return out, lse


@_forward_op.register_fake
def _forward_fake(query, key, value, mask, bias, scale, geometry, flags, want_lse):
    out = torch.empty_like(query)
    count = query.numel() // query.shape[-1] if want_lse else 0
    return out, query.new_empty((count,), dtype=torch.float32)


@torch.library.custom_op("oops_b200::triangle_attention_backward", mutates_args=())
def _backward_op(
    grad_out: Tensor, query: Tensor, key: Tensor, value: Tensor, mask: Optional[Tensor], bias: Optional[Tensor],
    out: Tensor, lse: Tensor, scale: float, geometry: List[int], flags: int, need: List[bool],
) -> Tuple[Tensor, Tensor, Tensor, Tensor]:
    given = (query, key, value, bias)
    grads = _reverse_of_saved(decode_geometry(geometry), grad_out, query, key, value, mask, bias, out, lse, scale, flags, need)
    empty = torch.empty(0, dtype=query.dtype, device=query.device)

    def laid_out_like(grad, operand):
        # the fake implementation promises the operand's own strides; a gradient computed on a re-laid copy
        # (unaligned or non-unit-stride operands) is copied into that layout
        if grad is None:
            return empty
        if operand is None or grad.stride() == operand.stride():
            return grad
        return torch.empty_like(operand).copy_(grad)

    return tuple(laid_out_like(g, operand) for g, operand in zip(grads, given))


@_backward_op.register_fake
def _backward_fake(grad_out, query, key, value, mask, bias, out, lse, scale, geometry, flags, need):
    def like(t, wanted):
        return torch.empty_like(t) if wanted and t is not None else query.new_empty((0,))

    return like(query, need[0]), like(key, need[1]), like(value, need[2]), like(bias, need[3])


def _dispatch_setup(ctx, inputs, output):
    query, key, value, mask, bias, scale, geometry, flags, _want = inputs
    out, lse = output
    ctx.save_for_backward(query, key, value, mask, bias, out, lse)
    ctx.scale, ctx.geometry, ctx.flags = scale, geometry, flags
    ctx.set_materialize_grads(False)


def _dispatch_backward(ctx, grad_out, _grad_lse):
    if grad_out is None:
        return (None,) * 9
    query, key, value, mask, bias, out, lse = ctx.saved_tensors
    need = [ctx.needs_input_grad[0], ctx.needs_input_grad[1], ctx.needs_input_grad[2],
            ctx.needs_input_grad[4] and bias is not None]
    dq, dk, dv, db = _backward_op(grad_out, query, key, value, mask, bias, out, lse, ctx.scale, ctx.geometry, ctx.flags, need)
    return (dq if need[0] else None, dk if need[1] else None, dv if need[2] else None, None, db if need[3] else None,
            None, None, None, None)


_forward_op.register_autograd(_dispatch_backward, setup_context=_dispatch_setup)


def _needs_dispatcher(*tensors: Optional[Tensor]) -> bool:
    if torch.compiler.is_compiling() or proxy_tracing():
        return True
    from torch._subclasses.fake_tensor import is_fake

    return any(t is not None and is_fake(t) for t in tensors)


def apply(query, key, value, mask, bias, scale, geometry, flags=0) -> Tensor:
    if _needs_dispatcher(query, key, value, mask, bias):
        want_lse = torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in (query, key, value, bias))
        out, _ = _forward_op(query, key, value, mask, bias, scale, encode_geometry(geometry), flags, want_lse)
        return out
    if torch._C._functorch.peek_interpreter_stack() is not None:
        raise unsupported("triangle_attention", "does not support torch.func transforms")
    if tracing():
        return TracedAttention.apply(query, key, value, mask, bias, float(scale), geometry, flags)
    return result_like(native().attend(query, key, value, mask, bias, scale, encode_geometry(geometry), flags), query)
