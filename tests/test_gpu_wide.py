"""The sweeps that share a particle among lanes, at the particle counts where
their width changes (32 lanes up to 5,550 particles, then 16, 8, 4, and one
thread past 44,400) and at the smallest ones, against the oracle bit for bit:
a random cloud with a clump of over a hundred mutual neighbours (several
rounds of staged hits) and coincident particles, a list cap that some
particles exceed (the same clump makes one long run of the grid's keys), and
two divergence and two density iterations, so every
sweep runs.
"""
import numpy as np
import pytest

from test_gpu_step import assert_same_bits, pair, same_state, step_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 33, 5550, 5551, 11101, 22201, 44401])
def test_lane_shared_sweeps_match_the_oracle(fcu, orc, n):
    d = 0.01
    side = max(4, round(n ** (1 / 3))) * d
    sim, o = pair(fcu, orc, geometry=fcu.GEOMETRY_BOX, box_lo=(0, 0, 0), box_hi=(side, side, side), spacing=d,
                  rest_density=1000.0, seeding=fcu.SEED_NONE, count=n, xsph_blend=0.01, nbr_cap=60,
                  div_iters=2, den_iters=2)
    rng = np.random.default_rng(n)
    pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0, side, (n, 3))
    m = min(n // 2, 130)
    pos[:m, :3] = 0.6 * side + rng.uniform(-0.004, 0.004, (m, 3))
    pos[: m // 20, :3] = pos[m // 20, :3]
    vel[:, :3] = rng.uniform(-0.5, 0.5, (n, 3))
    prev_p = rng.uniform(0, 2000, n).astype(np.float32)
    for s in (sim, o):
        s.set_state(pos4=pos, vel4=vel, prev_p=prev_p)
    s_g, s_o = step_pair(fcu, orc, force=(0.5, -9.81, 0.2), dt=5e-4, v_clamp=8.0, omega=(0.1, 0, 0.4))
    for _ in range(2):
        sim.step(s_g)
        o.substep(s_o, 2, 2)
    for f in ("starts", "perm", "density", "alpha", "nbr_n", "kd", "pressure", "accel", "xsph", "work_vel", "wall_grad", "counters"):
        assert_same_bits(sim.field(f), o.field(f), f)
    assert n < 300 or sim.field("counters")[1] > 0
    same_state(sim, o, f"{n} particles")
