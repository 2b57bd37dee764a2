"""The branch-free unit vector against sqrtf and the IEEE division, bit for bit: every significand of the squared length at
both parities of its exponent, every significand of the length with numerators at random and beside midpoints, and vectors
across the bounds of their range."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_sweep(cuda_lib, tmp_path):
    from tests import cuda_build
    out = (C.c_ulonglong * 5)()
    vectors = 1 << 24
    assert cuda_build.load("unit_vector", tmp_path).sweep(out, 64, vectors) == 0
    roots, reciprocals, quotients, wrong, taken = out
    assert (roots, reciprocals, quotients, wrong) == (0, 0, 0, 0)
    assert vectors // 4 < taken < vectors
