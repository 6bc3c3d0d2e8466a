"""What an adjoint handle holds on the device before its first backward, and
that a long schedule, which goes round the forward's few velocity buffers many
times, leaves the loss and the gradient what the backward's own tapes (a buffer
per iteration) make of it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = float(np.float32(1.0 / 120.0))


def handle(fcu, wl, block, frames, precision):
    hi = tuple(float(k) for k in np.array(block) * 0.01)
    cfg = wl.box_config(fcu, block, hi, 0.005, seed=7, xsph=0.01)
    dts = float(np.float32(DT) / np.float32(4))
    return fcu.Adjoint(cfg, frames, 4, DT, wl.v_clamp(0.005, dts), 1, precision=precision)


# with unpadded vectors and a velocity per iteration of the longest schedule
# 6,200 and 13,400 bytes a particle
@pytest.mark.parametrize("precision,most", [(32, 6200), (64, 13400)])
def test_bytes_a_particle(fcu, wl, precision, most):
    import torch
    torch.zeros(1, device="cuda")
    free = torch.cuda.mem_get_info()[0]
    a = handle(fcu, wl, (64, 32, 64), 1, precision)
    used = free - torch.cuda.mem_get_info()[0]
    print(f"{used / a.n:.0f} bytes a particle")
    assert 0 < used <= most * a.n


@pytest.mark.parametrize("div,den", [(1, 0), (2, 3), (7, 8), (126, 126)])
def test_long_schedules_keep_their_bits(fcu, wl, div, den):
    # the backward recomputes each segment into its own tapes, so a frozen
    # second forward must give the first one's loss, and the gradient must not
    # depend on how often the forward ran
    a = handle(fcu, wl, (16, 8, 16), 1, 32)
    a.set_schedule([div] * 4, [den] * 4)
    controls = ([[0.3, -9.81, 0.1]], 0.01, [0.05, 0.02, 0.05])
    loss = a.forward(*controls)
    p, v = a.final_state()
    g, gx = a.backward()
    assert np.isfinite(loss) and np.all(np.isfinite(v)) and np.all(np.isfinite(g))
    assert a.forward(*controls) == loss
    p2, v2 = a.final_state()
    assert np.array_equal(p, p2) and np.array_equal(v, v2)
    g2, gx2 = a.backward()
    assert np.array_equal(g.view(np.uint64), g2.view(np.uint64)) and gx == gx2
