"""What the adjoint does where it cannot answer: a bounded wait of its
neighbour grid that gives up (run out on purpose, as the simulations' tests
do; nothing faults and the handle stays usable) is reported by the forward
or the backward that used the grid.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = float(np.float32(1.0 / 120.0))


def small(fcu, wl, precision, frames=2, every=1):
    cfg = wl.box_config(fcu, (16, 8, 16), (0.32, 0.32, 0.32), 0.005, seed=7, xsph=0.01)
    dts = float(np.float32(DT) / np.float32(4))
    return fcu.Adjoint(cfg, frames, 4, DT, wl.v_clamp(0.005, dts), every, precision=precision)


CONTROLS = ([[0.3, -9.81, 0.1], [-0.2, -9.81, 0.4]], 0.01, [0.05, 0.02, 0.05])


@pytest.mark.parametrize("precision", [32, 64])
def test_a_grid_wait_that_gives_up_is_reported(fcu, wl, precision):
    a = small(fcu, wl, precision)
    loss = a.forward(*CONTROLS)
    grad, gx = a.backward()
    for call in (lambda: a.forward(*CONTROLS), a.backward):
        assert fcu.lib().fluid_selftest_adjoint_wait(a.h) == fcu.OK
        with pytest.raises(fcu.FluidError) as e:
            call()
        assert e.value.code == fcu.ERR_TIMEOUT and "gave up" in str(e.value)
        # reported once; the handle answers as before
        assert a.forward(*CONTROLS) == loss
    g2, gx2 = a.backward()
    assert np.array_equal(g2.view(np.uint64), grad.view(np.uint64)) and gx2 == gx


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("precision", [32, 64])
def test_a_state_that_is_no_number_is_refused(fcu, wl, precision, bad):
    # positions that are NaN all stand in one cell, each a neighbour of every
    # other: past the model's cap of 128
    a = small(fcu, wl, precision)
    forces, xsph, target = CONTROLS
    with pytest.raises(fcu.FluidError) as e:
        a.forward([forces[0], [0.0, bad, 0.0]], xsph, target)
    assert e.value.code == fcu.ERR_STATE and "128 neighbours" in str(e.value)
    assert np.isfinite(a.forward(*CONTROLS))
