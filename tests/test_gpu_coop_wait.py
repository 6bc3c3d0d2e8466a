"""The barrier of the one-launch grid build, run out on purpose without a
fault: a barrier that expects an arrival more than come. The kernel ends by
itself, nothing is written outside the outputs, the give-up is reported, and a
build and a step afterwards are right.
"""
import numpy as np
import pytest

from test_gpu_grid_coop import build
from test_gpu_step import frame_dt, pair, same_state, step_pair, v_clamp

pytestmark = pytest.mark.gpu


def test_the_barrier_gives_up_and_reports_a_timeout(fcu, orc):
    import torch
    rc, ms = fcu.selftest_coop_wait(0)
    assert rc == fcu.ERR_TIMEOUT, (rc, fcu.last_error())
    assert "fluid_grid_build_status reported it" in fcu.last_error()
    assert 0.0 < ms < 20000.0, ms
    print(f"bounded barriers gave up after {ms:.1f} ms")
    rng = np.random.default_rng(3)
    pos = np.zeros((5003, 4), np.float32)
    pos[:, :3] = rng.uniform(0, 16, (5003, 3))
    keys, _, perm = build(fcu, torch, torch.from_numpy(pos).cuda(), (16, 16, 16))
    assert np.array_equal(perm[:5003], np.argsort(keys[:5003], kind="stable"))
    sim, o = pair(fcu, orc)
    dt = frame_dt(1)
    st, ost = step_pair(fcu, orc, force=(0.0, -9.81, 0.0), dt=dt, v_clamp=v_clamp(sim.cfg.spacing, dt))
    sim.step(st)
    o.substep(ost, sim.cfg.div_iters, sim.cfg.den_iters)
    same_state(sim, o, "after the timeout")
