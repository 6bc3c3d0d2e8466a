"""What a program that uses this framework has it do, as cases that can be timed.

Five families, each through the public entry points of fluidcu.py:

  box      one box of fluid stepped by the convergence-driven solve
           (FLUID_SOLVE_TOLERANCE), read back once per video picture
  slab     the reference application's slab with its fixed schedule, tracers
           and thickness field, read back every frame
  batch    many boxes of uneven size stepped by the same launches, read back
           as a training program reads its observations
  adjoint  the loss of a tilt-control sequence and its gradients
  grid     the neighbour grid alone, on device buffers

A case is a dict of plain values. prepare() makes what the program holds
before the call from the seed alone; run() is one pass and returns what the
program reads; exact() is the same in 64 bits with plain torch, for the
cases where that is quick: an independent statement of the substep (and, by
torch's autograd, of its gradients).
"""
import importlib
import math

import numpy as np
import torch
import torch.utils.checkpoint

fcu = importlib.import_module("fluid-simulation-app_b200.fluidcu")
wl = importlib.import_module("fluid-simulation-app_b200.workloads")

F32 = np.float32
FRAME_DT = float(F32(1.0 / 120.0))
SLAB_EXTENT = (4.0 * 0.0357, 4.0 * 0.0774)
SLAB_DEPTH = 4.0 * 0.00765
EXACT_MAX_PARTICLES = 80000


def listed():
    return [
        # the reference application's own scene (1,620 particles): a display
        # frame with its tracers, everything read back; launches and latency
        dict(name="slab_app", family="slab", spacing=0.01, frames=1, tracers=500, field_w=32,
             field_h=64, spin=0.4),
        # the same slab at a phone's full picture: finer particles, the
        # thickness field at a quarter of the drawable per axis
        dict(name="slab_fine", family="slab", spacing=0.0031, frames=1, tracers=4096, field_w=295,
             field_h=639, spin=0.0),
        # the dam break of the workloads, one 1/30 s picture of 1/120 s frames,
        # the program setting its substeps (0 elsewhere: the reference's policy)
        dict(name="dam_break_16k", family="box", nx=32, ny=16, nz=32, room=2.0, spacing=0.01,
             frames=4, substeps=4, warm=0, tracers=0),
        # a mid-size box with odd counts: a preview of a production run
        dict(name="box_odd_150k", family="box", nx=67, ny=33, nz=69, room=2.0, spacing=0.005,
             frames=4, substeps=0, warm=2, tracers=1000),
        # the benchmark's million particles under the tilt, one picture
        dict(name="tilt_1m", family="box", nx=128, ny=64, nz=128, room=2.0, spacing=0.005,
             frames=2, substeps=0, warm=4, tracers=4096),
        # a small batch: few environments, one control step of two frames
        dict(name="batch_8", family="batch", boxes=8, lo=4096, hi=8192, frames=2, warm=1),
        # the batched workload's distribution of boxes, one such step
        dict(name="batch_64", family="batch", boxes=64, lo=4096, hi=65536, frames=2, warm=3),
        # a gradient step of the tilt-control problem on the adjoint box
        dict(name="adjoint_64k", family="adjoint", nx=64, ny=16, nz=64, frames=4, every=10,
             precision=32),
        # the double-precision gradient that finite differences are held to
        dict(name="adjoint_8k_f64", family="adjoint", nx=32, ny=8, nz=32, frames=2, every=1,
             precision=64),
        # the neighbour grid alone: a small cloud, an odd ordinary one
        # packed at the bottom of its box, and the 16.7M-position workload
        dict(name="grid_20k", family="grid", n=20011, side=24, kind="uniform"),
        dict(name="grid_1m_packed", family="grid", n=1000003, side=100, kind="packed"),
        dict(name="grid_16m", family="grid", n=1 << 24, side=256, kind="uniform"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["slab", "box", "batch", "adjoint", "grid", "box", "grid"])
    if kind == "slab":
        return dict(family="slab", spacing=round(_log(rng, 0.0031, 0.01), 5), frames=rng.randint(1, 2),
                    tracers=rng.choice([0, 500, 1777, 4096]), field_w=rng.randint(24, 295),
                    field_h=rng.randint(48, 639), spin=round(rng.uniform(0.0, 0.8), 3))
    if kind == "box":
        m = _log(rng, 8.0, 60.0)
        return dict(family="box", nx=max(4, int(2 * m * rng.uniform(0.9, 1.1))), ny=max(4, int(m)),
                    nz=max(4, int(2 * m * rng.uniform(0.9, 1.1))), room=round(rng.uniform(1.3, 2.0), 2),
                    spacing=rng.choice([0.005, 0.01]), frames=rng.randint(1, 2),
                    substeps=rng.choice([0, 0, 4, 8]), warm=rng.randint(0, 3),
                    tracers=rng.choice([0, 0, 1000, 4096]))
    if kind == "batch":
        hi = int(_log(rng, 6000, 65536))
        return dict(family="batch", boxes=int(_log(rng, 4, 64)), lo=4096, hi=hi, frames=rng.randint(1, 2),
                    warm=rng.randint(0, 3))
    if kind == "adjoint":
        m = rng.uniform(6.0, 16.0)
        return dict(family="adjoint", nx=int(4 * m), ny=max(4, int(m * rng.uniform(0.7, 1.0))), nz=int(4 * m),
                    frames=rng.randint(1, 4), every=rng.randint(1, 10), precision=rng.choice([32, 32, 64]))
    n = int(_log(rng, 2000, 1 << 24))
    return dict(family="grid", n=n, side=max(4, int((n / rng.uniform(0.8, 8.0)) ** (1.0 / 3.0))),
                kind=rng.choice(["uniform", "packed", "gaussian"]))


# ---- inputs --------------------------------------------------------------------


def _slab_state(case, seed):
    """Positions and velocities of the slab, half full and swirling."""
    d = case["spacing"]
    dims = [max(1, int(v / d + 1e-6)) for v in
            (2 * SLAB_EXTENT[0] - d, 0.5 * (2 * SLAB_EXTENT[1] - d), SLAB_DEPTH - d)]
    origin = np.array([-0.5 * dims[0] * d, -SLAB_EXTENT[1] + 0.5 * d, -0.5 * dims[2] * d])
    half = np.array([0.5, 0.0, 0.5])
    return _lattice(dims, origin + half * d, d, 0.1, 0.15, seed)


def _box_state(case, seed):
    d = case["spacing"]
    return _lattice((case["nx"], case["ny"], case["nz"]), np.full(3, 0.5 * d), d, 0.005, 0.3, seed)


def _lattice(dims, origin, d, jitter, speed, seed):
    """Lattice centres with a jitter, moving with a smooth random swirl."""
    rng = np.random.default_rng(seed)
    iz, iy, ix = np.meshgrid(*(np.arange(k) for k in reversed(dims)), indexing="ij")
    at = np.stack([ix, iy, iz], -1).reshape(-1, 3)
    pos = np.zeros((at.shape[0], 4), F32)
    pos[:, :3] = origin + at * d + rng.uniform(-jitter * d, jitter * d, at.shape)
    unit = at / np.maximum(np.array(dims) - 1, 1)
    vel = np.zeros_like(pos)
    for axis in range(3):
        for _ in range(2):
            k, phase = rng.uniform(1.0, 4.0, 3), rng.uniform(0, 2 * math.pi)
            vel[:, axis] += (0.5 * speed * np.sin(unit @ k + phase)).astype(F32)
    return pos, vel


def _tilt(seed, frames):
    return wl.tilt_schedule(1 + seed % 100003, frames, 1.0 / 120.0)


def _box_cfg(case, seed):
    d = case["spacing"]
    hi = tuple(float(F32(case["room"] * k * d)) for k in (case["nx"], case["ny"], case["nz"]))
    n = case["nx"] * case["ny"] * case["nz"]
    return wl.box_config(fcu, (1, 1, 1), hi, d, tracers=case["tracers"], seeding=fcu.SEED_NONE, count=n)


def _batch_cfgs(case, seed):
    cfgs = wl.batched_boxes(fcu, case["boxes"], lo=case["lo"], hi=case["hi"])
    for b, cfg in enumerate(cfgs):
        cfg.seed = 1 + seed * 100003 + b
    return cfgs


def _adjoint_hi(case):
    """Four block widths and eight block heights, as the adjoint workload."""
    return tuple(float(F32(w * k)) for k, w in ((case["nx"], 0.02), (case["ny"], 0.04), (case["nz"], 0.02)))


def _controls(case, seed):
    rng = np.random.default_rng(seed)
    forces = _tilt(seed, case["frames"]).astype(np.float64)
    span = np.array([case["nx"], case["ny"], case["nz"]]) * 0.005
    return forces, 0.01 * rng.uniform(0.5, 1.5), span * rng.uniform(0.4, 0.8, 3)


SUBSTEPS = 4  # of the adjoint's frames


def prepare(case, seed):
    fam = case["family"]
    s = dict(case=case, frame=0)
    if fam in ("box", "slab"):
        if fam == "box":
            s["sim"] = fcu.Sim(_box_cfg(case, seed))
            pos, vel = _box_state(case, seed)
        else:
            pos, vel = _slab_state(case, seed)
            s["sim"] = fcu.Sim(fcu.default_config(spacing=case["spacing"], seeding=fcu.SEED_NONE,
                                                  count=pos.shape[0], tracers=case["tracers"]))
        s["sim"].set_state(pos, vel)
        s["forces"] = _tilt(seed, 4096)
        for _ in range(case.get("warm", 0)):
            _frame(s)
    elif fam == "batch":
        s["batch"] = fcu.Batch(_batch_cfgs(case, seed))
        s["seed"], s["v_max"] = 1 + seed % 100003, [0.0] * case["boxes"]
        for _ in range(case["warm"]):
            _batch_frame(s)
    elif fam == "adjoint":
        cfg = wl.box_config(fcu, (case["nx"], case["ny"], case["nz"]), _adjoint_hi(case), 0.005,
                            seed=1 + seed % 100003)
        dts = float(F32(FRAME_DT) / F32(SUBSTEPS))
        s["adjoint"] = fcu.Adjoint(cfg, case["frames"], SUBSTEPS, FRAME_DT, wl.v_clamp(0.005, dts),
                                   case["every"], case["precision"])
        s["forces"], s["xsph"], s["target"] = _controls(case, seed)
    else:
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        n, side = case["n"], float(case["side"])
        pos = torch.zeros((n, 4), device="cuda")
        if case["kind"] == "gaussian":
            at = torch.rand((8, 3), generator=gen, device="cuda") * (side * 0.75) + side / 8
            which = torch.randint(0, 8, (n,), generator=gen, device="cuda")
            pos[:, :3] = at[which] + torch.randn((n, 3), generator=gen, device="cuda") * (side / 16)
        else:
            pos[:, :3] = torch.rand((n, 3), generator=gen, device="cuda") * side
            if case["kind"] == "packed":
                pos[: int(n * 0.9), 1] *= 0.1
        g = fcu.FluidGrid()
        g.cell = 1.0
        g.dims[:] = [case["side"]] * 3
        bytes_ = fcu.grid_workspace_bytes(n, g)
        s.update(pos=pos, grid=g, ws_bytes=bytes_, ws=torch.empty(bytes_, dtype=torch.uint8, device="cuda"),
                 starts=torch.empty(case["side"] ** 3 + 1, dtype=torch.int32, device="cuda"),
                 perm=torch.empty(n, dtype=torch.int32, device="cuda"))
    return s


# ---- passes --------------------------------------------------------------------


def _frame(s):
    """One 1/120 s frame, and its telemetry."""
    sim, k = s["sim"], s["frame"]
    spin = s["case"].get("spin", 0.0)
    sim.frame(tuple(float(v) for v in s["forces"][k % len(s["forces"])]), FRAME_DT,
              omega=(0.0, 0.0, spin), domega=(0.0, 0.0, 0.5 * spin),
              substeps=s["case"].get("substeps", 0), seed=k)
    s["frame"] = k + 1
    return sim.stats()


def _batch_frame(s):
    """One frame of every box on the shared substep clock, and the boxes' statistics."""
    batch, k = s["batch"], s["frame"]
    n = max(fcu.substeps_for(FRAME_DT, v, wl.BATCH_SPACING, 16) for v in s["v_max"])
    batch.run(wl.batched_frame_steps(fcu, batch.nboxes, 1, n, s["seed"], k))
    batch.reduce_stats()
    stats = batch.stats()
    s["frame"], s["v_max"] = k + 1, [t.v_max for t in stats]
    return stats


def run(s):
    case = s["case"]
    if case["family"] in ("box", "slab"):
        sim = s["sim"]
        for _ in range(case["frames"]):
            stats = _frame(s)
        pos, vel = sim.read_particles()
        out = dict(pos=pos, vel=vel, stats=stats.as_reference_block())
        if case["tracers"]:
            out["tracers"] = sim.tracers()
        if case["family"] == "slab":
            sim.field_splat(case["field_w"], case["field_h"], keep=0.6, lens=4, lo=0.0, hi=0.5)
            sim.field_filter()
            out["field"], out["filtered"] = sim.field_read()
        return out
    if case["family"] == "batch":
        for _ in range(case["frames"]):
            stats = _batch_frame(s)
        states = [s["batch"].state(b) for b in range(s["batch"].nboxes)]
        out = {k: np.concatenate([x[k] for x in states]) for k in ("pos", "vel", "id")}
        out["stats"] = np.stack([t.as_reference_block() for t in stats])
        return out
    if case["family"] == "adjoint":
        adj, real = s["adjoint"], F32 if case["precision"] == 32 else np.float64
        loss = adj.forward(s["forces"], s["xsph"], s["target"])
        pos, vel = adj.final_state()
        grad, grad_xsph = adj.backward()
        # a program with 32-bit controls keeps their gradients in 32 bits
        return dict(loss=real(loss), grad=grad.astype(real), grad_xsph=real(grad_xsph),
                    pos=pos.astype(real), vel=vel.astype(real))
    fcu.grid_build_device(s["pos"].data_ptr(), case["n"], s["grid"], 0, s["starts"].data_ptr(),
                          s["perm"].data_ptr(), s["ws"].data_ptr(), s["ws_bytes"],
                          torch.cuda.current_stream().cuda_stream)
    return dict(starts=s["starts"], perm=s["perm"])


def _particles(case):
    if case["family"] == "slab":
        return _slab_state(case, 0)[0].shape[0]
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Bytes: each record of a substep's sweeps read and written once, each
    output once. Flops: the pair terms (about 33 pairs a particle in the
    splashing fluid; 60 flops in the density sweep, 80 in the forces, 20 in
    each of the other sweeps)."""
    fam = case["family"]
    if fam == "grid":
        return dict(bytes=16.0 * case["n"] + 4.0 * case["n"] + 4.0 * case["side"] ** 3, flops=0.0)
    if fam == "batch":
        # counts log-uniform in [lo, hi]
        lo, hi = case["lo"], case["hi"]
        n = case["boxes"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)
        sub = 12 * case["frames"]
    elif fam == "adjoint":
        n, sub = _particles(case), SUBSTEPS * case["frames"]
        real = 4 if case["precision"] == 32 else 8
        # the forward, its recomputation and the reverse sweeps
        return dict(bytes=3.0 * n * sub * 100 * real, flops=4.0 * n * sub * 33 * 220)
    else:
        n = _particles(case)
        sub = case["frames"] * (12 if fam == "box" else 8)
    pairs = 33.0 * n * sub
    out = 32.0 * n + (24.0 * case["field_w"] * case["field_h"] if fam == "slab" else 0.0)
    return dict(bytes=612.0 * n * sub + out, flops=pairs * (60 + 80 + 4 * 20))


# ---- the same in 64 bits ---------------------------------------------------------

# Boundary polynomials of the reference (sim_solve.wgsl:249-293): coefficient
# [i][j] of t1^i t2^j.
WEDGE = [
    [2.5005807e-01, -3.4681153e-01, -4.0986882e-02, 3.0301620e-01, -1.9202736e-01, 4.6947582e-02, -3.8543515e-03],
    [-3.4681153e-01, 4.8587248e-01, 1.0092180e-02, -2.9978363e-01, 1.5320335e-01, -2.2544282e-02],
    [-4.0986882e-02, 1.0092180e-02, -5.4145610e-02, 7.9597369e-02, -2.3350373e-02],
    [3.0301620e-01, -2.9978363e-01, 7.9597369e-02, -8.2431946e-03],
    [-1.9202736e-01, 1.5320335e-01, -2.3350373e-02],
    [4.6947582e-02, -2.2544282e-02],
    [-3.8543515e-03],
]
WEDGE_D = [
    [-3.4611994e-01, 4.4757673e-01, 1.1932939e-01, -4.6460101e-01, 2.7637253e-01, -6.2846025e-02, 4.3871652e-03],
    [-6.3622823e-02, 2.0521006e-01, -3.7311339e-01, 3.7508155e-01, -1.6629713e-01, 2.5030129e-02],
    [7.8352497e-01, -1.2658344e+00, 5.8898945e-01, -1.0772903e-01, 1.3535777e-02],
    [-4.9470084e-01, 9.1302071e-01, -3.4330355e-01, 2.4034609e-02],
    [-2.5605481e-02, -2.0067981e-01, 5.9854468e-02],
    [8.8898623e-02, 3.9914838e-03],
    [-1.7788321e-02],
]


def _poly2(table, t1, t2):
    out = torch.zeros_like(t1)
    for row in reversed(table):
        inner = torch.zeros_like(t1)
        for c in reversed(row):
            inner = inner * t2 + c
        out = out * t1 + inner
    return torch.where(t1 * t1 + t2 * t2 >= 4.0, torch.zeros_like(out), out)


def _wall_density(t):
    near = 0.5 - 0.7 * t + t**3 / 3 - 0.15 * t**5 + 0.05 * t**6
    far = 8 / 15 - 0.8 * t + 2 / 3 * t**3 - 0.5 * t**4 + 0.15 * t**5 - t**6 / 60
    return torch.where(t >= 2, torch.zeros_like(t), torch.where(t < 1, near, far))


def _wall_gradient(t):
    near = 0.7 - t**2 + 0.75 * t**4 - 0.3 * t**5
    far = 0.8 - 2 * t**2 + 2 * t**3 - 0.75 * t**4 + 0.1 * t**5
    return torch.where(t >= 2, torch.zeros_like(t), torch.where(t < 1, near, far))


def _wall_adhesion(t):
    u = (2.0 - t).clamp(0.0, 2.0)
    return u * u * (1.7847015e-3 + u * (3.3392196e-3 + u * (-4.3394677e-3 + u * (1.6711868e-3 - u * 2.1788750e-4))))


class _Fluid:
    """The substep in float64 (sim_solve.wgsl), particles in their own order."""

    def __init__(self, spacing, rho0, lo, hi, xsph, div=(0.01, 1), den=(0.001, 0), tolerance=True, max_iters=100):
        self.h = float(F32(1.2) * F32(spacing))
        d = F32(spacing)
        self.rho0, self.m = float(F32(rho0)), float(F32(rho0) * d * d * d)
        self.lo, self.hi = (torch.tensor([float(F32(v)) for v in w], dtype=torch.float64, device="cuda") for w in (lo, hi))
        h = F32(self.h)
        self.sigma = float(F32(1) / (F32(math.pi) * h * h * h))
        self.xsph, self.div, self.den, self.tolerance, self.max_iters = xsph, div, den, tolerance, max_iters
        self.counts = None  # frozen iteration counts of the substeps, when kept

    def pairs(self, x):
        """Every ordered pair within the support."""
        sup = 2.0 * self.h
        with torch.no_grad():
            axis = int((x.max(0).values - x.min(0).values).argmax())
            order = torch.argsort(x[:, axis])
            y = x[order].contiguous()
            key = y[:, axis].contiguous()
            out = []
            for a in range(0, y.shape[0], 2048):
                b = min(a + 2048, y.shape[0])
                c0 = int(torch.searchsorted(key, key[a] - sup))
                c1 = int(torch.searchsorted(key, key[b - 1] + sup, right=True))
                d2 = torch.zeros((b - a, c1 - c0), dtype=torch.float64, device=x.device)
                for k in range(3):
                    d2 += (y[a:b, None, k] - y[None, c0:c1, k]) ** 2
                i, j = torch.nonzero(d2 < 4.0 * self.h * self.h, as_tuple=True)
                i, j = i + a, j + c0
                keep = i != j
                out.append(torch.stack([order[i[keep]], order[j[keep]]]))
            return torch.cat(out, 1)

    def kernel(self, r):
        """W and its derivative."""
        q = r / self.h
        near = 1 - 1.5 * q * q * (1 - 0.5 * q)
        t = 2 - q
        w = self.sigma * torch.where(q < 1, near, 0.25 * t**3)
        dw = self.sigma / self.h * torch.where(q < 1, -3 * q + 2.25 * q * q, -0.75 * t * t)
        return w, dw

    def walls(self, x):
        tl, th = (x - self.lo) / self.h, (self.hi - x) / self.h
        t = torch.cat([tl, th], 1)  # x y z low, then high
        fill = _wall_density(t).sum(1)
        for a, b in ((0, 1), (0, 2), (1, 2)):
            for ka in (a, a + 3):
                for kb in (b, b + 3):
                    fill = fill - _poly2(WEDGE, t[:, ka], t[:, kb])
        grad = []
        for a in range(3):
            g = torch.zeros_like(fill)
            for ka, sign in ((a, -1.0), (a + 3, 1.0)):
                s = _wall_gradient(t[:, ka])
                for kb in range(6):
                    if kb % 3 != a:
                        s = s + _poly2(WEDGE_D, t[:, ka], t[:, kb])
                g = g + sign * s
            grad.append(self.rho0 / self.h * g)
        adh = _wall_adhesion(th) - _wall_adhesion(tl)
        return fill, torch.stack(grad, 1), adh

    def density(self, x):
        n = x.shape[0]
        i, j = self.pairs(x)
        e = x[i] - x[j]
        r = e.square().sum(1).sqrt()
        w, dw = self.kernel(r)
        gw = (dw / r)[:, None] * e
        fold = lambda v: torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device).index_add(0, i, v)  # noqa: E731
        fill, wg, adh = self.walls(x)
        rho = self.m * (fold(w) + self.sigma) + self.rho0 * fill
        near = fold((1 - r / self.h).clamp(min=0.0) ** 3)
        big = self.m * fold(gw) + wg
        alpha = rho / (big.square().sum(1) + self.m**2 * fold(gw.square().sum(1))).clamp(min=1e-4)
        return dict(i=i, j=j, e=e, r=r, w=w, gw=gw, fold=fold, wg=wg, adh=adh, rho=rho, near=near, alpha=alpha)

    def substep(self, st, dt, v_clamp, force, omega=None, domega=None, k=None):
        x, v, pp, temp = st["x"], st["v"], st["pp"], st["temp"]
        D = self.density(x)
        i, j, e, r, gw, fold, wg, rho = (D[q] for q in ("i", "j", "e", "r", "gw", "fold", "wg", "rho"))
        m, rho0 = self.m, self.rho0
        diverge = lambda v: m * fold(((v[i] - v[j]) * gw).sum(1)) + (v * wg).sum(1)  # noqa: E731
        push = lambda v, kd: v - dt * (m * fold((kd[i] + kd[j])[:, None] * gw) + kd[:, None] * wg)  # noqa: E731
        frozen = self.counts[k] if self.counts is not None and k is not None and k < len(self.counts) else None

        def loop(which, tol, fixed):
            nonlocal v, pressure
            it = 0
            while True:
                d = diverge(v)
                if which == 0:
                    res, kd = d.clamp(min=0.0) * dt / rho0, d.clamp(min=0.0) * D["alpha"] / dt / rho
                else:
                    over = (rho + dt * d - rho0).clamp(min=0.0)
                    res, kd = over / rho0, over * D["alpha"] / (dt * dt) / rho
                if frozen is not None:
                    go = it < frozen[which]
                elif self.tolerance:
                    go = it < self.max_iters and (float(res.detach().mean()) > tol or (which == 0 and it < 1))
                else:
                    go = it < fixed
                if not go:
                    return it
                v = push(v, kd)
                if which == 1:
                    pressure = pressure + kd * rho * rho
                it += 1

        pressure = 0.5 * pp
        n_div = loop(0, *self.div)
        # forces
        dv = v[i] - v[j]
        pair = m / (rho[i] * rho[j]) * (e * gw).sum(1) / (r * r + 0.01 * self.h**2)
        c = 2.0 * self.h
        coh = (c - r) ** 3 * r**3
        coh = torch.where(2 * r > c, coh, 2 * coh - c**6 / 64) * 32.0 / (math.pi * c**9)
        sig = 0.0728
        gamma = sig * 7040.0 / (21.0 * 0.8665 * rho0 * rho0 * c * c)
        beta = sig * (1.0 - 0.342) * 1558.4 / (0.8665 * rho0 * rho0 * c * c)
        near = fold(((D["near"][i] + D["near"][j]) * (1 - r / self.h).clamp(min=0.0) ** 2 / r)[:, None] * e)
        tension = -fold((2 * rho0 / (rho[i] + rho[j]) * m * coh / r)[:, None] * e)
        visc = fold((2 * 1.002e-3 * pair)[:, None] * dv)
        blend = -fold((m / rho[j] * D["w"])[:, None] * dv)
        acc = visc + 3000.0 * near + gamma * tension + beta * rho0 * D["adh"]
        if temp is not None:
            heat = 2 * 0.598 / 4184.0 * pair * (temp[i] - temp[j])
            heat = fold(heat - 0.5 * 1.002e-3 / 4184.0 * pair * dv.square().sum(1))
            temp = temp + dt * heat
        blend_k = self.xsph if torch.is_tensor(self.xsph) or self.xsph >= 0 else 1.0 - math.exp(-6.0 * dt)
        a = acc + force
        if omega is not None:
            w_, dw_ = omega.expand_as(x), domega.expand_as(x)
            cr = torch.linalg.cross
            a = a - cr(dw_, x) - cr(w_, cr(w_, x)) - 2.0 * cr(w_, v)
        v = push(v + dt * a + blend_k * blend, 0.5 * pp / (rho * rho))
        n_den = loop(1, *self.den)
        if self.counts is not None and frozen is None:
            self.counts.append((n_div, n_den))
        # integrate
        speed = v.square().sum(1).clamp(min=1e-60).sqrt()
        ceiling = torch.where(rho < 0.5 * rho0, 3.0 * v_clamp, v_clamp)
        fast = speed > ceiling
        v = torch.where(fast[:, None], v * (ceiling / speed)[:, None], v)
        to = x + v * dt
        at = torch.minimum(torch.maximum(to, self.lo), self.hi)
        out = dict(x=at, pp=pressure, temp=temp)
        out["v"] = out["pv"] = torch.where(at == to, v, torch.zeros_like(v))
        if "accel" in st:
            chase = 1.0 - math.exp(-20.0 * dt)
            accel = (v - st["pv"]).square().sum(1).sqrt() / dt
            out["accel"] = st["accel"] * (1 - chase) + accel * chase
            out["lens"] = st["lens"] * (1 - chase) + pressure * chase
            out["temp"] = temp + temp * 2.07e-4 / (rho * 4184.0) * (pressure - pp)
        return out


def _f64(a):
    return torch.as_tensor(a, device="cuda").double()


def _exact_sim(case, seed):
    slab = case["family"] == "slab"
    pos, vel = (_slab_state if slab else _box_state)(case, seed)
    d, n = case["spacing"], pos.shape[0]
    if slab:
        ext = SLAB_EXTENT + (SLAB_DEPTH / 2,)
        fl = _Fluid(d, 998.2, [-v for v in ext], ext, -1.0, tolerance=False)
    else:
        hi = [case["room"] * k * d for k in (case["nx"], case["ny"], case["nz"])]
        fl = _Fluid(d, 1000.0, (0.0, 0.0, 0.0), hi, float(F32(0.01)))
    zero = torch.zeros(n, dtype=torch.float64, device="cuda")
    st = dict(x=_f64(pos[:, :3]), v=_f64(vel[:, :3]), pp=zero, temp=zero + float(F32(293.15)), accel=zero, lens=zero)
    st["pv"] = torch.zeros_like(st["v"])  # set_state leaves the velocity of the substep before at zero
    forces = _tilt(seed, 4096)
    spin = torch.tensor([0.0, 0.0, float(F32(case.get("spin", 0.0)))], dtype=torch.float64, device="cuda")
    for k in range(case.get("warm", 0) + case["frames"]):
        # by the policy (render.rs:57-106) a first frame runs its floor, or
        # eight cheaper substeps where the floor is over 0.65 of that
        floor = min(8, math.ceil(FRAME_DT / (0.42 * d) - 1e-6))
        sub = case.get("substeps", 0) or (8 if floor > 5 else floor)
        dt = float(F32(FRAME_DT) / F32(sub))
        vc = float(F32(0.4) * F32(d) / F32(dt))
        fl.den = (0.001, 5 if dt > 0.00105 else 2)
        for _ in range(sub):
            st = fl.substep(st, dt, vc, _f64(forces[k]), spin, 0.5 * spin)
    out = dict(pos=torch.cat([st["x"], zero[:, None]], 1).cpu().numpy(),
               vel=torch.cat([st["v"], st["accel"][:, None]], 1).cpu().numpy(), stats=None)
    if case["tracers"]:
        out["tracers"] = None
    if slab:
        out["field"], out["filtered"] = _exact_field(case, fl, st)
    return out


def _exact_field(case, fl, st):
    """The splat of every particle over an empty field, blended at 0.4, and the filter."""
    W, H = case["field_w"], case["field_h"]
    ex, ey = SLAB_EXTENT
    x, y = st["x"][:, 0] / ex, st["x"][:, 1] / ey
    rx, ry = 1.5 * fl.h / ex, 1.5 * fl.h / ey
    lens = (st["v"].square().sum(1).sqrt() / 0.5).clamp(0.0, 1.0)
    tx0 = ((x - rx + 1) * 0.5 * W - 0.5).floor().long() - 1
    ty0 = ((1 - (y + ry)) * 0.5 * H - 0.5).floor().long() - 1
    field = torch.zeros((2, H * W), dtype=torch.float64, device="cuda")
    for oy in range(int(ry * H) + 5):
        ty = ty0 + oy
        cy = (1 - (ty + 0.5) / H * 2 - y) / ry
        for ox in range(int(rx * W) + 5):
            tx = tx0 + ox
            cx = ((tx + 0.5) / W * 2 - 1 - x) / rx
            w = (1 - cx * cx - cy * cy).clamp(min=0.0) ** 2 * 0.5
            ok = (tx >= 0) & (tx < W) & (ty >= 0) & (ty < H) & (w > 0)
            at = (ty * W + tx)[ok]
            field[0].index_add_(0, at, w[ok])
            field[1].index_add_(0, at, (w * lens)[ok])
    field = (0.4 * field).reshape(2, H, W)
    taps = torch.tensor([0.015625, 0.09375, 0.234375, 0.3125, 0.234375, 0.09375, 0.015625], dtype=torch.float64, device="cuda")
    pad = torch.nn.functional.pad(field[None, :1], (4, 4, 4, 4), mode="replicate")
    blur = torch.nn.functional.conv2d(pad, taps.reshape(1, 1, 1, 7))
    blur = torch.nn.functional.conv2d(blur, taps.reshape(1, 1, 7, 1))[0, 0]
    c = blur[1:-1, 1:-1]
    xp, xm, yp, ym = blur[1:-1, 2:], blur[1:-1, :-2], blur[2:, 1:-1], blur[:-2, 1:-1]
    aspect = (ex / W) ** 2 / (ey / H) ** 2
    filtered = torch.stack([c, xp - xm, ym - yp, (xp + xm - 2 * c) + (yp + ym - 2 * c) * aspect], -1)
    return field.permute(1, 2, 0).cpu().numpy(), filtered.cpu().numpy()


def _exact_adjoint(case, seed):
    """The model's loss and its gradients by autograd, each substep recomputed in the backward."""
    d = 0.005
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    # the lattice block's jitter: a splitmix64 stream over x, y, z of each particle
    n = nx * ny * nz
    with np.errstate(over="ignore"):
        z = np.uint64(1 + seed % 100003) + np.uint64(0x9E3779B97F4A7C15) * np.arange(1, 3 * n + 1, dtype=np.uint64)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    u = ((z >> np.uint64(40)).astype(F32) * F32(1.0 / 16777216.0)).reshape(n, 3)
    iz, iy, ix = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    at = np.stack([ix, iy, iz], -1).reshape(n, 3).astype(F32)
    amp = F32(0.005) * F32(d)
    x0 = (at + F32(0.5)) * F32(d) + (F32(2) * u - F32(1)) * amp
    forces, xsph, target = _controls(case, seed)
    f = _f64(forces).requires_grad_(True)
    c = torch.tensor(xsph, dtype=torch.float64, device="cuda", requires_grad=True)
    fl = _Fluid(d, 1000.0, (0.0, 0.0, 0.0), _adjoint_hi(case), c)
    fl.counts = []
    dt = float(F32(FRAME_DT) / F32(SUBSTEPS))
    vc = wl.v_clamp(d, dt)

    def step(x, v, pp, force, cc, k):
        fl.xsph = cc
        out = fl.substep(dict(x=x, v=v, pp=pp, temp=None), dt, vc, force, k=k)
        return out["x"], out["v"], out["pp"]

    x = _f64(x0)
    v, pp = torch.zeros_like(x), torch.zeros(n, dtype=torch.float64, device="cuda")
    for k in range(case["frames"] * SUBSTEPS):
        x, v, pp = torch.utils.checkpoint.checkpoint(step, x, v, pp, f[k // SUBSTEPS], c, k, use_reentrant=False)
    rho = torch.utils.checkpoint.checkpoint(lambda y: fl.density(y)["rho"], x, use_reentrant=False)
    loss = (x.mean(0) - _f64(target)).square().sum() + (rho / 1000.0 - 1.0).square().mean()
    loss.backward()
    h = lambda t: t.detach().cpu().numpy()  # noqa: E731
    return dict(loss=h(loss), grad=h(f.grad), grad_xsph=h(c.grad), pos=h(x), vel=h(v))


def exact(case, seed):
    fam = case["family"]
    if fam in ("box", "slab"):
        frames = case.get("warm", 0) + case["frames"]
        # later frames of the policy's count hang on a speed's last bits (its ceil)
        known = frames == 1 or (case.get("substeps", 0) > 0 and frames <= 4)
        return _exact_sim(case, seed) if known and _particles(case) <= EXACT_MAX_PARTICLES else None
    if fam == "adjoint":
        return _exact_adjoint(case, seed)
    return None  # a batch and the large boxes take too long; the grid's outputs are whole numbers
