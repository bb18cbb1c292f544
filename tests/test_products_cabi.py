"""Which lists of products the C entry point serves: operands that an epilogue needs and does not get, rows that overlap or run backwards, unknown
epilogues and counts are refused on the host, with no launch."""

import ctypes
from ctypes import Structure, c_int32, c_int64, c_void_p

import pytest

from oops_b200.runtime import cabi

PLAIN, GATE, REVERSE = 0, 1, 2


class Product(Structure):
    _fields_ = [("a", c_void_p), ("a_ld", c_int64), ("b", c_void_p), ("b_ld", c_int64), ("c", c_void_p), ("c_ld", c_int64),
                ("m", c_int32), ("n", c_int32), ("k", c_int32), ("a_transposed", c_int32), ("b_transposed", c_int32), ("epilogue", c_int32),
                ("values", cabi.Pair), ("dvalues", cabi.Pair), ("gate", c_void_p), ("gate_ld", c_int64), ("gated", c_void_p), ("gated_ld", c_int64),
                ("tokens", c_int32), ("dim", c_int32)]


def product(kind=PLAIN, **over):
    pair = cabi.Pair(0x40000, 64 * 32, 0, 32, 8)
    p = Product(a=0x10000, a_ld=40, b=0x20000, b_ld=40, c=0x30000, c_ld=32, m=100, n=32, k=40, epilogue=kind)
    if kind != PLAIN:
        p.values, p.gate, p.gate_ld, p.gated, p.gated_ld, p.tokens, p.dim = pair, 0x50000, 32, 0x60000, 32, 64, 8
    if kind == REVERSE:
        p.dvalues, p.c = pair, None
    for key, value in over.items():
        setattr(p, key, value)
    return p


def supported(*items, dtype=cabi.BF16, count=None):
    lib = cabi.library()
    array = (Product * max(1, len(items)))(*items)
    return lib.oops_ta_products_supported(dtype, ctypes.byref(array), len(items) if count is None else count)


def test_what_is_served():
    for epilogue in (PLAIN, GATE, REVERSE):
        assert supported(product(epilogue)) == 1 and supported(product(epilogue), dtype=cabi.F16) == 1
    assert supported(product(GATE), product(REVERSE)) == 1
    assert supported(product(a_transposed=1, a_ld=104, b_transposed=1, b_ld=32)) == 1
    assert supported(product(REVERSE, gated=None)) == 1 and supported(product(REVERSE, dvalues=cabi.Pair())) == 1


REFUSED = [(PLAIN, dict(a=None)), (PLAIN, dict(b=None)), (PLAIN, dict(c=None)), (GATE, dict(c=None)), (GATE, dict(values=cabi.Pair())),
           (GATE, dict(gated=None)), (REVERSE, dict(values=cabi.Pair())), (REVERSE, dict(gate=None)), (PLAIN, dict(c_ld=24)),
           (PLAIN, dict(c_ld=-32)), (GATE, dict(gated_ld=24)), (GATE, dict(gated_ld=-32)), (REVERSE, dict(gate_ld=24)),
           (REVERSE, dict(gated_ld=8)), (PLAIN, dict(a_ld=32)), (PLAIN, dict(b_ld=-40)), (PLAIN, dict(a_transposed=1, a_ld=96)),
           (PLAIN, dict(epilogue=3)), (GATE, dict(epilogue=7)), (PLAIN, dict(epilogue=-1)), (PLAIN, dict(a=0x10002)), (PLAIN, dict(c=0x30008)),
           (PLAIN, dict(n=28)), (PLAIN, dict(m=0)), (PLAIN, dict(k=-8)), (PLAIN, dict(m=2**31 - 1)), (GATE, dict(tokens=0)), (GATE, dict(dim=12)),
           (GATE, dict(values=cabi.Pair(0x40008, 2048, 0, 32, 8))), (REVERSE, dict(dvalues=cabi.Pair(0x40000, 2048, 0, 33, 8)))]


@pytest.mark.parametrize("epilogue,over", REFUSED)
def test_what_is_refused(epilogue, over):
    assert supported(product(epilogue, **over)) == 0
    assert supported(product(), product(epilogue, **over)) == 0


def test_counts_and_types():
    assert supported(product(), count=0) == 0 and supported(product(), count=-1) == 0
    assert supported(product(), count=3) == 0  # (more than a launch takes: the list is not walked)
    assert supported(product(), dtype=cabi.F32) == 0
    assert cabi.library().oops_ta_products_supported(cabi.BF16, None, 1) == 0


@pytest.mark.gpu
def test_refused_lists_launch_nothing(cuda):
    lib = cabi.library()
    before = cabi.launch_count()
    for epilogue, over in REFUSED:
        assert lib.oops_ta_products(cabi.BF16, ctypes.byref(product(epilogue, **over)), 1, None) != 0
    assert lib.oops_ta_products(cabi.BF16, None, 1, None) != 0 and lib.oops_ta_products(cabi.BF16, ctypes.byref(product()), 0, None) != 0
    assert cabi.launch_count() == before
