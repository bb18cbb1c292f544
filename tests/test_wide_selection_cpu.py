"""Which calls of a head size other than 32 take the tcgen05 kernels for them: served types and layouts, and the sizes at which they are the faster
ones (as measured: the rule's own comment has the times)."""

from __future__ import annotations

import ctypes

import pytest

from oops_b200.runtime import cabi


def problem(rows, cols, heads, dim, **over):
    p = cabi.Problem()
    p.abi_version, p.dtype, p.bias_dtype = cabi.ABI_VERSION, cabi.BF16, cabi.BF16
    p.batch, p.rows, p.cols, p.heads, p.head_dim, p.scale = 1, rows, cols, heads, dim, 1.0
    for name in ("q", "k", "v"):
        setattr(p, name, pair(p))
    width = (cols + 7) // 8 * 8
    p.bias_groups, p.bias, p.bias_sk, p.bias_sq, p.bias_sh = 1, 0x20000, 1, width, cols * width
    p.bias_sg = p.bias_sb = heads * cols * width
    for key, value in over.items():
        setattr(p, key, value)
    return p


def pair(p):
    return cabi.Pair(0x10000, p.rows * p.cols * p.heads * p.head_dim, p.cols * p.heads * p.head_dim, p.heads * p.head_dim, p.head_dim)


def forward(p, out=None):
    return cabi.library().oops_ta_uses_wide_path(ctypes.byref(p), ctypes.byref(out or pair(p)), None)


def reverse(p, want):
    g = cabi.Grads()
    for name in "qkv":
        if name in want:
            setattr(g, "d" + name, pair(p))
    if "b" in want:
        g.dbias = 0x30000
    return cabi.library().oops_ta_uses_wide_path(ctypes.byref(p), ctypes.byref(pair(p)), ctypes.byref(g))


def test_types_and_layouts():
    assert forward(problem(4, 512, 16, 64)) == 1 and reverse(problem(4, 512, 16, 64), "qkvb") == 1
    assert forward(problem(4, 512, 16, 64, dtype=cabi.F16, bias_dtype=cabi.F16)) == 0
    assert forward(problem(4, 512, 16, 64, mask=0x40000)) == 0 and forward(problem(4, 512, 16, 64, bias_dtype=cabi.F32)) == 0
    assert forward(problem(4, 512, 16, 32)) == 0 and forward(problem(4, 512, 16, 72)) == 0 and forward(problem(4, 512, 16, 60)) == 0
    assert forward(problem(4, 512, 16, 64, bias=0x20008)) == 0 and forward(problem(4, 512, 16, 64, bias_sq=516)) == 0
    assert forward(problem(4, 512, 16, 64, flags=cabi.FLAG_FORCE_GENERIC)) == 0
    p = problem(4, 512, 16, 64)
    p.k.sc = 0
    assert forward(p) == 0
    p = problem(4, 512, 16, 64)
    out = pair(p)
    out.ptr = 0x10002
    assert forward(p, out) == 0
    assert cabi.library().oops_ta_uses_wide_path(ctypes.byref(p), None, None) == -cabi.STATUS_INVALID_ARGUMENT


@pytest.mark.parametrize("rows,cols,heads,dim,taken", [(1, 64, 16, 64, 0), (1, 65, 16, 64, 1), (1, 85, 8, 48, 0), (1, 86, 8, 48, 1), (1, 128, 8, 24, 0),
                                                       (1, 129, 8, 24, 1), (96, 256, 4, 16, 0), (96, 257, 4, 8, 1), (1, 300, 8, 16, 0),
                                                       (1, 384, 8, 8, 1)])
def test_forward_sizes(rows, cols, heads, dim, taken):
    assert forward(problem(rows, cols, heads, dim)) == taken


@pytest.mark.parametrize("rows,cols,heads,dim,taken", [
    # taken for: (all gradients, without the bias's, queries alone)
    (1024, 64, 4, 64, (1, 0, 0)), (37, 64, 4, 64, (1, 1, 1)), (1024, 64, 4, 16, (0, 0, 0)), (1, 64, 8, 16, (1, 0, 0)), (2048, 8, 4, 24, (1, 0, 0)),
    (1, 65, 8, 48, (1, 1, 1)), (256, 160, 4, 40, (1, 1, 1)), (1, 192, 8, 24, (1, 0, 0)), (18, 128, 4, 24, (1, 1, 1)), (1, 256, 8, 24, (1, 1, 1)),
    (256, 160, 4, 8, (0, 0, 0)), (256, 160, 4, 16, (1, 0, 0)), (256, 128, 4, 16, (1, 1, 1)), (256, 193, 4, 16, (1, 1, 1)), (1, 256, 8, 16, (0, 0, 0)),
    (1, 384, 8, 16, (1, 0, 0)), (7, 300, 4, 16, (1, 1, 0))])
def test_reverse_sizes(rows, cols, heads, dim, taken):
    p = problem(rows, cols, heads, dim)
    assert (reverse(p, "qkvb"), reverse(p, "qkv"), reverse(p, "q")) == taken
    assert reverse(p, "b") == 1  # (the bias gradient alone)
