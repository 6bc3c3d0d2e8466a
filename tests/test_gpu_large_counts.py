"""The one-thread sweeps, which run above 44,400 particles, against the oracle
bit for bit: batches whose total stands on either side of every change of the
sweeps' width (5,550, 11,100, 22,200 and 44,400 particles), uneven boxes that
stop their loops on their own, every block size and the autotuner above the
last; and one box above it with a stencil row longer than 4,096 slots, with
positions on the slab and cell edges, with a large neighbour cap, and with
coordinates next to the coordinate planes.
"""
import numpy as np
import pytest

from test_gpu_batch import oracle_twin, same_box, to_oracle_step
from test_gpu_slabs import edge_positions
from test_gpu_step import assert_same_bits, pair, same_state, step_pair, v_clamp

pytestmark = pytest.mark.gpu
F32 = np.float32

# totals 5,550, 5,551, 11,101, 22,201, 44,400 and 44,401
BOXES = [((15, 14, 15), (5, 5, 5), (7, 13, 25)), ((15, 14, 15), (5, 5, 9), (8, 16, 17)),
         ((19, 18, 19), (5, 5, 7), (9, 12, 41)), ((24, 22, 23), (5, 5, 16), (9, 29, 37)),
         ((28, 26, 30), (5, 5, 8), (20, 26, 43)), ((28, 26, 30), (5, 5, 7), (21, 26, 41))]
PAST = BOXES[-1]


def configs(fcu, wl, lattices, **kw):
    return [wl.box_config(fcu, lat, tuple(float(F32(0.01 * k)) for k in lat), 0.005, seed=31 + b,
                          xsph=0.005 + 0.01 * b, **kw) for b, lat in enumerate(lattices)]


@pytest.mark.parametrize("lattices", BOXES, ids=lambda l: str(sum(a * b * c for a, b, c in l)))
def test_batches_around_the_widths_match_the_oracle(fcu, orc, wl, lattices):
    nb = len(lattices)
    steps = wl.batched_frame_steps(fcu, nb, frames=2, substeps=2, seed=8)
    batch = fcu.Batch(configs(fcu, wl, lattices, den_tol=0.0002))
    twins = [oracle_twin(orc, batch, b) for b in range(nb)]
    seen = set()
    for k, row in enumerate(steps):
        batch.step(row)
        stats = batch.stats()
        for b in range(nb):
            iters, res = twins[b].substep_tol(to_oracle_step(orc, row[b]), 0.01, 0.0002, 100)
            assert (stats[b].div_iters, stats[b].den_iters) == (int(iters[0]), int(iters[1])), (k, b)
            assert stats[b].div_residual == res[0] and stats[b].den_residual == res[1], (k, b)
        seen.add(tuple(t.den_iters for t in stats))
    for b in range(nb):
        same_box(batch, twins[b], b, "tolerance")
    assert any(len(set(row)) > 1 for row in seen)  # the boxes stop at different iterations
    fixed = fcu.Batch(configs(fcu, wl, lattices, solve=fcu.SOLVE_FIXED, div_iters=2, den_iters=2))
    twins = [oracle_twin(orc, fixed, b) for b in range(nb)]
    fixed.run(steps[:2])
    for row in steps[:2]:
        for b in range(nb):
            twins[b].substep(to_oracle_step(orc, row[b]), 2, 2)
    for b in range(nb):
        same_box(fixed, twins[b], b, "fixed")


@pytest.mark.parametrize("kw", [dict(), dict(solve=1, div_iters=2, den_iters=2)])
def test_block_sizes_change_no_bit_past_the_last_width(fcu, wl, kw):
    if kw:
        kw["solve"] = fcu.SOLVE_FIXED
    nb = len(PAST)
    cfgs = configs(fcu, wl, PAST, **kw)
    steps = wl.batched_frame_steps(fcu, nb, frames=2, substeps=3, seed=9)
    ref = fcu.Batch(cfgs)
    ref.run(steps)
    want = [ref.state(b) for b in range(nb)]

    def same(batch, what):
        for b in range(nb):
            got = batch.state(b)
            for k in want[b]:
                assert_same_bits(got[k], want[b][k], f"{what} box {b} {k}")

    for tpb in (64, 128, 256):
        other = fcu.Batch(cfgs)
        other.set_blocks([tpb] * 7)
        other.run(steps)
        same(other, f"{tpb} threads")
    tuned = fcu.Batch(cfgs)
    tuned.run(steps[:2])
    chosen, ms = tuned.autotune(steps[2])
    assert set(chosen.values()) <= {64, 128, 256} and np.all(ms > 0)
    tuned.run(steps[2:])
    same(tuned, f"tuned {chosen}")


def box(fcu, orc, n, side, **kw):
    cfg = dict(geometry=fcu.GEOMETRY_BOX, box_lo=(0, 0, 0), box_hi=(side, side, side), spacing=0.01,
               h_ratio=1.0, rest_density=1000.0, seeding=fcu.SEED_NONE, count=n, xsph_blend=0.01,
               div_iters=2, den_iters=2)
    cfg.update(kw)
    return pair(fcu, orc, **cfg)


def run_both(fcu, orc, sim, o, pos, vel=None, dt=5e-4):
    for s in (sim, o):
        s.set_state(pos4=pos, vel4=vel)
    s_g, s_o = step_pair(fcu, orc, force=(0.4, -9.81, 0.2), dt=dt, v_clamp=v_clamp(0.01, dt))
    sim.step(s_g)
    o.substep(s_o, 2, 2)
    for f in ("starts", "perm", "density", "alpha", "nbr_n", "kd", "pressure", "accel", "xsph", "counters"):
        assert_same_bits(sim.field(f), o.field(f), f)
    same_state(sim, o)


def test_a_stencil_row_past_4096_slots(fcu, orc):
    n = 45001
    sim, o = box(fcu, orc, n, 0.36)
    rng = np.random.default_rng(12)
    pos = np.zeros((n, 4), F32)
    pos[:, :3] = rng.uniform(0, 0.36, (n, 3))
    at = rng.permutation(n)[:4500]
    p = sim.params  # at a cell's centre, so that one row of cells holds all of it
    centre = np.array(p.box_min, F32) + F32(p.cell) * F32(9.5)
    pos[at, :3] = centre + rng.uniform(-0.004, 0.004, (4500, 3)).astype(F32)
    pos[at[:10], :3] = pos[at[10], :3]  # exact duplicates: r = 0 pairs
    run_both(fcu, orc, sim, o, pos, dt=1e-4)
    starts, d = sim.field("starts").astype(np.int64), p.dims
    cell = (9 * d[1] + 9) * d[0] + 9
    assert starts[4 * (cell + 1)] - starts[4 * cell] > 4096
    assert sim.field("counters")[1] > 0 and sim.field("nbr_n").max() == sim.cfg.nbr_cap


@pytest.mark.parametrize("kw", [dict(h_ratio=1.2), dict(h_ratio=1.2, nbr_cap=300)])
def test_slab_edges_and_a_large_cap(fcu, orc, kw):
    n = 44999
    sim, o = box(fcu, orc, n, 0.36, **kw)
    run_both(fcu, orc, sim, o, edge_positions(sim.params, n, 3))


# Where a particle stands within 2^-36 of a coordinate plane its pairs divide
# as written, elsewhere six quotients share one reciprocal: both in one cloud.
@pytest.mark.parametrize("n", [3001, 45003])
def test_coordinates_next_to_the_planes(fcu, orc, n):
    half = 0.5 * max(4, round(n ** (1 / 3))) * 0.01
    sim, o = box(fcu, orc, n, half, box_lo=(-half, -half, -half))
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4), F32)
    pos[:, :3] = rng.uniform(-half, half, (n, 3))
    near = np.array([0.0, -0.0, 1e-45, -1e-38, 1e-30, -1e-20, 2.0**-60, 2.0**-37, -(2.0**-36), 2.0**-36 * 1.5, 1e-9], F32)
    for axis in range(3):
        at = rng.permutation(n)[: n // 4]
        pos[at, axis] = rng.choice(near, at.size)
    vel = np.zeros((n, 4), F32)
    vel[:, :3] = rng.uniform(-0.5, 0.5, (n, 3))
    run_both(fcu, orc, sim, o, pos, vel)
