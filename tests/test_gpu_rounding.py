"""The square root and the quotient of the packed perception against CUDA's correctly rounded ones."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_root_and_quotient_equal_the_rounded_intrinsics():
    """Every mantissa of two neighbouring binades (an even and an odd exponent), 2^17 of each other binade from 2^-66 to 2^66; per
    root one quotient, its numerator a random mantissa and 2^-40 to 2^40 times the root."""
    from npa_b200 import _native as n
    wrong = torch.zeros(2, dtype=torch.int32, device="cuda")
    total = 0
    for exponent in range(-66, 66):
        count, step = (1 << 23, 1) if exponent in (-4, -3) else (1 << 17, 61)      # an odd step: all residues of the low bits
        n.check(n.lib.npa_rounding_selftest((exponent + 127) << 23, step, count, exponent + 1000, n.ptr(wrong), n.current_stream()))
        total += count
    assert wrong.tolist() == [0, 0], f"of {total} roots and quotients {wrong.tolist()} differ"


def test_operands_outside_the_range_are_refused():
    from npa_b200 import _native as n
    wrong = torch.full((2,), 7, dtype=torch.int32, device="cuda")
    for first, step, count in ((1, 1, 10), (((127 + 66) << 23) - 5, 1, 10), ((127 - 67) << 23, 1, 1)):
        rc = n.lib.npa_rounding_selftest(first, step, count, 0, n.ptr(wrong), n.current_stream())
        assert rc == n.NPA_ERR_INVALID_ARGUMENT and wrong.tolist() == [7, 7]
