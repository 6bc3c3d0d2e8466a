"""The forces' quotients by a shared reciprocal are the correctly rounded ones:
random operands over the ranges a pair brings (the host refuses none of them),
with significands of all zeros and all ones among them.
"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 2])
def test_quotients_are_the_divisions(fcu, seed):
    differ = C.c_uint64(1)
    assert fcu.lib().fluid_selftest_quotient(0, seed, 1 << 31, C.byref(differ)) == fcu.OK
    assert differ.value == 0
