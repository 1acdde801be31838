"""The smoother's own square root, reciprocal and divisions are the correctly
rounded ones: every significand of two binades and a stride of the rest for the
root and its reciprocal, whose exceptions the residual flags and nothing else;
quotients at and beside the half-way points of subnormal results, with powers of
two and any divisor, and of every size."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_pd_math(cuda):
    from cvt_gb300 import _lib
    bad = (ctypes.c_ulonglong * 4)(*[9] * 4)
    assert _lib.lib().cvtpm_tool_pd_math_check(0, None, bad) == 0
    assert list(bad) == [0, 0, 0, 0]
    assert _lib.lib().cvtpm_tool_pd_math_check(0, None, None) != 0
