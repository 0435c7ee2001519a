"""The separately rounded kernels' division and square root (integer remainders, no FP64 instructions)
against the hardware's IEEE ones: on log-uniform operands, on raw bit patterns (subnormal, zero,
infinite and NaN included) and on nearly equal significands.  They have to be equal: the self-test counts
any difference as 2^20 units in the last place, and the fast build's own error is at most 2."""
import ctypes as C

import pytest

from mhdturbulence_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,seed", [(1, 7), (4097, 8), (1 << 22, 9), (1 << 24, 10)])
def test_division_and_root_equal_ieee(n, seed):
    m = C.c_double()
    assert _lib.lib().mhdgb_selftest_division(0, n, seed, C.byref(m)) == 0
    assert m.value <= 2.0, m.value
