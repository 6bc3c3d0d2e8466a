"""The adjoint model's density sweep at its three widths (8 lanes a particle up
to 37,888 particles, then 4, one thread from 177,600 in 32 bits and 325,600 in
64): the same lists, scales, densities and wall gradients to the bit, for the
smallest counts, ragged ones, and one past every change of width.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = float(np.float32(1.0 / 120.0))


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("block", [(1, 1, 1), (3, 1, 1), (13, 7, 11), (35, 19, 57), (65, 49, 63), (71, 67, 69)])
def test_the_widths_agree(fcu, wl, block, precision):
    hi = tuple(max(0.04, k * 0.01) for k in block)
    cfg = wl.box_config(fcu, block, hi, 0.005, seed=7, xsph=0.01)
    a = fcu.Adjoint(cfg, 1, 2, DT, wl.v_clamp(0.005, 0.5 * DT), 1, precision=precision)
    assert a.n == block[0] * block[1] * block[2]
    a.forward([[0.3, -9.81, 0.1]], 0.01, [0.1, 0.05, 0.1])
    differ = C.c_uint64(1)
    assert fcu.lib().fluid_selftest_adjoint_density(a.h, C.byref(differ)) == fcu.OK
    assert differ.value == 0
    with pytest.raises(fcu.FluidError):  # its forward's densities are gone
        a.backward()
