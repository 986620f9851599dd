"""Timed cases of the framework: what its users have it do, through its public
entry points, over the range of sizes, shape orders, precisions and boundary
kinds that the repository's configurations and tests use.

A pass is what a program does between two outputs: a number of loop steps,
then the arrays (and, in the restart cases, the particles) on the host; in the
adjoint cases one evaluation of an objective with its gradient.

kinds
  thermal   periodic (or absorbing-x) thermal plasma: `steps` loop steps, then
            every field, current and charge array
  laser     a laser pulse in an underdense plasma, absorbing faces, 4th order:
            `steps` loop steps of a run that has the pulse inside, then the
            arrays
  observed  the same plasma watched: after every loop step the diagnostics
            (energies, charge, Gauss residual), the arrays at the end
  restart   particle records from the host, `steps` loop steps, particle
            records back to the host, in the order of their ids
  adjoint   kinetic energy in a window after `steps` steps, and its gradient
            with respect to every particle's weight and the laser's amplitude
            coefficients; `segment` steps per checkpoint
"""
import math

import numpy as np
import torch

PI = 3.1415926536            # the value of pi every derived length of the framework uses
LAMBDA = 2.0 * PI
FIELDS = ("ex", "ey", "ez", "bx", "by", "bz")
RINGS = ("jx", "jy", "jz", "rho0", "rho1")
MASS = (1.0, 1836.0)
CHARGE = (-1.0, 1.0)


def listed():
    return [
        # the smallest grid the parity tests use: launches and latency
        dict(name="restart_12x10x11_o4_fp64", kind="restart", nx=12, ny=10, nz=11, order=4, prec="fp64", ppc0=1,
             ppc1=1, u=0.1, per_x=1, steps=4),
        # the 32^3 thermal plasma, 8 electrons per cell over a fixed background, in both precisions
        dict(name="thermal_32_o2_fp64", kind="thermal", nx=32, ny=32, nz=32, order=2, prec="fp64", ppc0=8, ppc1=0,
             u=0.05, per_x=1, steps=20),
        # a ragged box with absorbing x faces (particles leave), few particles per cell
        dict(name="thermal_45x38x51_o2_fp32", kind="thermal", nx=45, ny=38, nz=51, order=2, prec="fp32", ppc0=4,
             ppc1=4, u=0.1, per_x=0, steps=20),
        # a watched run: diagnostics after every step
        dict(name="observed_64_o2_fp64", kind="observed", nx=64, ny=64, nz=64, order=2, prec="fp64", ppc0=8, ppc1=8,
             u=0.02, per_x=1, steps=16),
        # the throughput configuration (8 + 8 per cell, u_th 0.02) at three sizes, both orders and precisions
        dict(name="thermal_128x64x64_o2_fp32", kind="thermal", nx=128, ny=64, nz=64, order=2, prec="fp32", ppc0=8,
             ppc1=8, u=0.02, per_x=1, steps=32),
        dict(name="thermal_128x64x64_o4_fp64", kind="thermal", nx=128, ny=64, nz=64, order=4, prec="fp64", ppc0=8,
             ppc1=8, u=0.02, per_x=1, steps=16),
        dict(name="thermal_131x69x62_o4_fp32", kind="thermal", nx=131, ny=69, nz=62, order=4, prec="fp32", ppc0=8,
             ppc1=8, u=0.02, per_x=1, steps=16),
        dict(name="thermal_256x128x128_o2_fp64", kind="thermal", nx=256, ny=128, nz=128, order=2, prec="fp64", ppc0=8,
             ppc1=8, u=0.02, per_x=1, steps=16),
        # the laser configuration on a quarter-length box, relativistic electrons
        dict(name="laser_80x48x48_o4_fp64", kind="laser", nx=80, ny=48, nz=48, order=4, prec="fp64", ppc0=8, ppc1=8,
             u=0.0, per_x=0, steps=16),
        dict(name="laser_96x48x56_o4_fp32", kind="laser", nx=96, ny=48, nz=56, order=4, prec="fp32", ppc0=8, ppc1=8,
             u=0.0, per_x=0, steps=32),
        # the differentiable run: one recorded segment (FP32), and segments recomputed from checkpoints (FP64)
        dict(name="adjoint_48x32x32_fp32", kind="adjoint", nx=48, ny=32, nz=32, order=4, prec="fp32", ppc0=8, ppc1=0,
             u=0.0, per_x=0, steps=24, segment=24),
        dict(name="adjoint_32x24x24_fp64", kind="adjoint", nx=32, ny=24, nz=24, order=4, prec="fp64", ppc0=8, ppc1=0,
             u=0.0, per_x=0, steps=18, segment=6),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["thermal", "thermal", "thermal", "laser", "laser", "observed", "restart", "adjoint"])
    prec = rng.choice(["fp64", "fp32"])
    c = dict(kind=kind, prec=prec, order=rng.choice([2, 4]), per_x=1, u=round(rng.uniform(0.01, 0.1), 4))
    if kind == "restart":
        c.update(nx=size(10, 32), ny=size(10, 28), nz=size(10, 28), ppc0=rng.choice([1, 2, 4]), steps=rng.randint(1, 8))
        c["ppc1"] = rng.choice([0, c["ppc0"]])
    elif kind == "adjoint":
        c.update(nx=size(16, 56), ny=size(12, 32), nz=size(12, 32), ppc0=rng.choice([4, 8]), ppc1=0, u=0.0, per_x=0,
                 order=4, steps=rng.randint(10, 24))
        c["segment"] = rng.choice([c["steps"], rng.randint(4, 9)])
    elif kind == "laser":
        c.update(nx=size(40, 112), ny=size(24, 56), nz=size(24, 56), ppc0=8, ppc1=8, u=0.0, per_x=0, order=4,
                 steps=rng.randint(4, 6) * 4)
    else:
        c.update(nx=size(12, 160), ny=size(12, 96), nz=size(12, 96), ppc0=rng.choice([1, 2, 4, 8, 8, 12]),
                 steps=rng.randint(3, 8) * 4)
        c["ppc1"] = rng.choice([0, c["ppc0"], c["ppc0"]])
        if kind == "thermal":
            c["per_x"] = rng.choice([1, 1, 1, 0])
    return c


# ---------------------------------------------------------------------------
# inputs


def _workload(case, seed):
    from pic3d_b200.workloads import Workload
    mem = 2 if case["order"] == 2 else 4
    grid = dict(name=case["kind"], nx=case["nx"], ny=case["ny"], nz=case["nz"], mem=mem,
                ppc=(case["ppc0"], case["ppc1"]), u_th=(case["u"], case["u"]), precision=case["prec"],
                steps=case["steps"])
    if case["kind"] == "laser":
        return Workload(period=(0, 0, 0), dx=LAMBDA / 20, dy=LAMBDA / 10, dz=LAMBDA / 10, absorbing=1,
                        laser_amplitude=2.0, laser_pulse_duration=10.0 * LAMBDA, laser_envelope=1,
                        laser_start_time=-10.0 * LAMBDA, waist=8.0 * LAMBDA, phase=0.1 * (seed % 7), **grid)
    if case["kind"] == "adjoint":
        return Workload(period=(0, 0, 0), dx=LAMBDA / 16, dy=LAMBDA / 16, dz=LAMBDA / 16, density_value=0.02,
                        laser_amplitude=1.0, laser_pulse_duration=10.0 * LAMBDA, waist=2.0 * LAMBDA, **grid)
    return Workload(period=(case["per_x"], 1, 1), **grid)


def _from_records(case):
    """Whether the particles come from host records (random positions of a
    numpy generator) or from the framework's device generator."""
    return case["kind"] in ("laser", "restart") or case["nx"] * case["ny"] * case["nz"] * case["ppc0"] <= 60000


def _particles(case, seed, kind):
    """Positions (cells), momenta and weights of one species."""
    ppc = case["ppc%d" % kind]
    n = case["nx"] * case["ny"] * case["nz"] * ppc
    rng = np.random.default_rng([seed, kind])
    c = np.repeat(np.arange(n // ppc if ppc else 0), ppc)
    x = rng.random((n, 3))
    x[:, 0] += c % case["nx"]
    x[:, 1] += (c // case["nx"]) % case["ny"]
    x[:, 2] += c // (case["nx"] * case["ny"])
    if case["u"] > 0:
        p = rng.normal(0.0, case["u"], (n, 3))
    else:
        p = np.zeros((n, 3))
    w = np.full(n, 1.0 / max(ppc, 1))
    if case["kind"] == "laser":
        w = 0.01 * np.minimum(1.0, x[:, 0] * (LAMBDA / 20) / (20 * LAMBDA)) / ppc
    return x, p, w


def _records(case, seed, kind):
    from pic3d_b200.workloads import PARTICLE_DTYPE
    x, p, w = _particles(case, seed, kind)
    r = np.zeros(len(w), dtype=PARTICLE_DTYPE)
    r["id"] = np.arange(len(w))
    r["x"], r["y"], r["z"] = x[:, 0], x[:, 1], x[:, 2]
    r["px"], r["py"], r["pz"] = p[:, 0], p[:, 1], p[:, 2]
    r["gamma"] = np.sqrt(1.0 + (p * p).sum(1))
    r["charge"], r["mass"], r["weight"] = CHARGE[kind], MASS[kind], w
    return r


def _pulse(case, seed):
    """ey and bz of a pulse inside the box: a carrier of unit wavelength in x
    under a smooth envelope, amplitude 2."""
    nx, m = case["nx"], 4
    i = np.arange(nx + 2 * m) - (m - 1.0)
    ph = 0.1 * (seed % 7)
    env = np.where((i > 0) & (i < 0.8 * nx), np.sin(np.pi * np.clip(i, 0, 0.8 * nx) / (0.8 * nx)) ** 2, 0.0)
    ihalf = i + 0.5
    envh = np.where((ihalf > 0) & (ihalf < 0.8 * nx), np.sin(np.pi * np.clip(ihalf, 0, 0.8 * nx) / (0.8 * nx)) ** 2, 0.0)
    ey = 2.0 * env * np.cos(2 * np.pi * i / 20 + ph)
    bz = 2.0 * envh * np.cos(2 * np.pi * ihalf / 20 + ph)
    shape = (case["nz"] + 2 * m, case["ny"] + 2 * m, nx + 2 * m)
    out = []
    for a in (ey, bz):
        full = np.zeros(shape)
        full[m:-m, m:-m, m:-m] = a[m:-m]
        out.append(full)
    return out


LASER_WARM = 8    # steps of the laser run before the timed ones


def prepare(case, seed):
    from pic3d_b200.simulation import Simulation
    w = _workload(case, seed)
    if case["kind"] == "adjoint":
        from pic3d_b200 import adjoint
        spec, knots, coef = _adjoint_problem(case, seed)
        run = adjoint.AdjointRun(spec, knots, coef)
        run._ck(run.lib.pic_checkpoint_save(run.ctx, 0))   # the initial state, for the next evaluation
        return dict(case=case, run=run)
    sim = Simulation(w, precision=case["prec"])
    state = dict(case=case, sim=sim)
    if case["kind"] == "restart":
        state["records"] = [_records(case, seed, k) for k in range(2)]
        return state
    for k in range(2):
        if case["ppc%d" % k]:
            if _from_records(case):
                sim.upload_particles(k, _records(case, seed, k))
            else:
                sim.generate_thermal(k, case["ppc%d" % k], 1.0, case["u"], seed + k)
    if case["kind"] == "laser":
        ey, bz = _pulse(case, seed)
        sim.upload_array("ey", ey)
        sim.upload_array("bz", bz)
    sim.initial_push()
    if case["kind"] == "laser":
        sim.run_main_time_loop(LASER_WARM)
    sim.synchronize()
    return state


def _adjoint_problem(case, seed):
    from pic3d_b200 import adjoint
    knots, coef = _adjoint_inputs(seed)
    spec = adjoint.AdjointSpec(workload=_workload(case, seed), n_knots=32, profile_n=8, window=_window(case),
                               ramp=2.0, segment=case["segment"], seed=seed, precision=case["prec"])
    return spec, knots, coef


def _adjoint_inputs(seed):
    rng = np.random.default_rng(seed)
    return 0.02 * (0.8 + 0.4 * rng.random(32)), 0.8 + 0.4 * rng.random((8, 8))


def _window(case):
    return (0.0, float(min(16, case["nx"])))


# ---------------------------------------------------------------------------
# passes


def _arrays(sim):
    """Every field, current and charge array on the host, in the run's precision."""
    out = {}
    for n in FIELDS + RINGS:
        a = torch.from_numpy(sim.download_array(n))
        out[n] = a.to(torch.float32) if sim.fp32 else a
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "adjoint":
        return _run_adjoint(case, state["run"])
    sim = state["sim"]
    if case["kind"] == "restart":
        zero_f, zero_r = np.zeros(sim.field_shape()), np.zeros(sim.ring_shape())
        for n in FIELDS:
            sim.upload_array(n, zero_f)
        for n in RINGS:
            sim.upload_array(n, zero_r)
        for k in range(2):
            sim.upload_particles(k, state["records"][k])
        sim.step = 0
        sim.initial_push()
        sim.run_main_time_loop(case["steps"])
        out = _arrays(sim)
        for k in range(2):
            r = sim.download_particles(k)
            r = r[np.argsort(r["id"])]
            for f in ("x", "y", "z", "px", "py", "pz", "weight"):
                out["%s%d" % (f, k)] = r[f].astype(np.float32) if sim.fp32 else r[f].copy()
        return out
    if case["kind"] == "observed":
        seen = []
        for _ in range(case["steps"]):
            sim.run_main_time_loop(1)
            d = sim.diagnostics()
            seen.append([d[k] for k in ("field_energy", "kinetic0", "kinetic1", "charge0", "charge1")])
        out = _arrays(sim)
        seen = np.array(seen)
        out["seen"] = seen.astype(np.float32) if sim.fp32 else seen
        return out
    sim.run_main_time_loop(case["steps"])
    return _arrays(sim)


def _run_adjoint(case, run):
    run._ck(run.lib.pic_checkpoint_restore(run.ctx, 0))
    run.bounds = []
    loss = run.forward()
    gw, gp = run.backward()
    if case["prec"] == "fp32":
        gw, gp = gw.astype(np.float32), gp.astype(np.float32)
    return {"loss": loss, "weights": gw, "profile": gp}


def work(case):
    cells = case["nx"] * case["ny"] * case["nz"]
    n = cells * (case["ppc0"] + case["ppc1"])
    f32 = case["prec"] == "fp32"
    real = 4 if f32 else 8
    # one push: a particle's position, momentum and weight read, position and
    # momentum written; gather of six components, current of three
    per_particle, per_cell = (60 if f32 else 104), 39 * real
    flops = 1100 if case["order"] == 2 else 3600
    pushes = case["steps"]
    extra = 11 * cells * 8
    if case["kind"] == "restart":
        pushes += 1
        extra += 2 * 144 * n + 11 * cells * 8
    if case["kind"] == "adjoint":
        # forward with its record, then the reverse sweep: the record and the
        # particle adjoints read and written, twice the forward's arithmetic
        pushes = (pushes + 1) * 3
        extra = n * 8
    return {"bytes": pushes * (n * per_particle + cells * per_cell) + extra, "flops": pushes * n * flops}


# ---------------------------------------------------------------------------
# the same loop in 64 bits with plain torch operations


def exact(case, seed):
    n = case["nx"] * case["ny"] * case["nz"] * (case["ppc0"] + case["ppc1"])
    steps = case["steps"] + (LASER_WARM if case["kind"] == "laser" else 0)
    cost = n * steps * (1.0 if case["order"] == 2 else 4.0) * (4.0 if case["kind"] == "adjoint" else 1.0)
    if cost > 6.0e8 or (not torch.cuda.is_available() and cost > 6.0e6):
        return None
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    loop = _Loop(case, seed)
    for k in range(2):
        loop.add_species(k, *_initial(case, seed, k))
    if case["kind"] == "laser":
        ey, bz = _pulse(case, seed)
        loop.f["ey"], loop.f["bz"] = loop.t(ey), loop.t(bz)
    loop.push()
    seen = []
    for s in range(1, steps + 1):
        loop.one_step(s)
        if case["kind"] == "observed":
            seen.append(loop.diagnostics())
    out = {k: v.cpu() for k, v in list(loop.f.items()) + list(loop.r.items())}
    if case["kind"] == "observed":
        out["seen"] = np.array(seen)
    if case["kind"] == "restart":
        for k in range(2):
            x, p, w = loop.sp[k]
            for d, f in enumerate("xyz"):
                out["%s%d" % (f, k)] = x[:, d].cpu()
                out["p%s%d" % (f, k)] = p[:, d].cpu()
            out["weight%d" % k] = w.cpu()
    return out


def _initial(case, seed, kind):
    if _from_records(case):
        return _particles(case, seed, kind)
    ppc = case["ppc%d" % kind]
    n = case["nx"] * case["ny"] * case["nz"] * ppc
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    q = torch.arange(n, device=dev, dtype=torch.int64)
    if n == 0:
        z = torch.zeros((0, 3), dtype=torch.float64, device=dev)
        return z, z, z[:, 0]
    # Philox4x32-10 (Salmon et al., SC 2011), key (seed, kind), counters (q, 0) and (q, 1)
    s = seed + kind
    key = (s & 0xFFFFFFFF, (s >> 32) ^ ((0x9E3779B9 * (kind + 1)) & 0xFFFFFFFF))
    u = []
    for h in range(2):
        u += _philox([q & 0xFFFFFFFF, q >> 32, torch.full_like(q, h), torch.zeros_like(q)], *key)
    u = [v.double() for v in u]
    t = 2.0 ** -32
    c = q // ppc
    x = torch.stack([(c % case["nx"]).double() + u[0] * t, ((c // case["nx"]) % case["ny"]).double() + u[1] * t,
                     (c // (case["nx"] * case["ny"])).double() + u[2] * t], 1)
    r0, r1 = torch.sqrt(-2 * torch.log((u[3] + 1) * t)), torch.sqrt(-2 * torch.log((u[5] + 1) * t))
    a0, a1 = 2 * math.pi * u[4] * t, 2 * math.pi * u[6] * t
    p = case["u"] * torch.stack([r0 * torch.cos(a0), r0 * torch.sin(a0), r1 * torch.cos(a1)], 1)
    return x, p, torch.full((n,), 1.0 / ppc, dtype=torch.float64, device=dev)


def _philox(c, k0, k1):
    def mul(a, b):   # 32 x 32 -> (high, low), in parts that fit 63 bits
        lo = a * (b & 0xFFFF)
        hi = a * (b >> 16) + (lo >> 16)
        return hi >> 16, ((hi & 0xFFFF) << 16) | (lo & 0xFFFF)

    for _ in range(10):
        h0, l0 = mul(c[0], 0xD2511F53)
        h1, l1 = mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _weights(d, order):
    """B-spline shape of the offset d from the nearest point, (N, order + 1)."""
    if order == 2:
        return torch.stack([0.5 * (0.5 - d) ** 2, 0.75 - d * d, 0.5 * (0.5 + d) ** 2], 1)

    def mid(u):
        return -u ** 4 / 6 + 5 * u ** 3 / 6 - 5 * u ** 2 / 4 + 5 * u / 24 + 55.0 / 96

    return torch.stack([(d - 0.5) ** 4 / 24, mid(1 + d), d ** 4 / 4 - 5 * d ** 2 / 8 + 115.0 / 192, mid(1 - d),
                        (d + 0.5) ** 4 / 24], 1)


class _Loop:
    """The per-timestep loop, straight from its formulas."""

    CHUNK = 1 << 20

    def __init__(self, case, seed, coef=None):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.order = case["order"]
        self.m = 2 if self.order == 2 else 4
        self.n = (case["nx"], case["ny"], case["nz"])
        laser, adj = case["kind"] == "laser", case["kind"] == "adjoint"
        self.per = (0, 0, 0) if laser or adj else (case["per_x"], 1, 1)
        self.d = (LAMBDA / 20, LAMBDA / 10, LAMBDA / 10) if laser else (LAMBDA / 16,) * 3 if adj else (1.0, 1.0, 1.0)
        self.dt = 0.95 / math.sqrt(sum(1.0 / h ** 2 for h in self.d))
        self.absorbing = laser
        self.amp = 2.0 if laser else 1.0 if adj else 0.0
        self.start = -10.0 * LAMBDA if laser else 0.0
        self.waist = 8.0 * LAMBDA if laser else 2.0 * LAMBDA
        self.phase = 0.1 * (seed % 7) if laser else 0.0
        self.coef = coef
        m = self.m
        fs = tuple(self.n[d] + 2 * m for d in (2, 1, 0))
        rs = tuple(s + 2 for s in fs)
        self.f = {k: torch.zeros(fs, dtype=torch.float64, device=self.dev) for k in FIELDS}
        self.r = {k: torch.zeros(rs, dtype=torch.float64, device=self.dev) for k in RINGS}
        self.sp = [None, None]

    def t(self, a):
        return torch.as_tensor(a, dtype=torch.float64, device=self.dev)

    def add_species(self, k, x, p, w):
        self.sp[k] = (self.t(x), self.t(p), self.t(w))

    # -- fields ------------------------------------------------------------
    def _in(self, a, dz=0, dy=0, dx=0, ring=0):
        m = self.m + ring
        nx, ny, nz = self.n
        return a[m + dz:m + dz + nz, m + dy:m + dy + ny, m + dx:m + dx + nx]

    def _add(self, name, v):
        """a physical-cell increment of a field, then its periodic ghosts"""
        m = self.m
        a = self.f[name] + torch.nn.functional.pad(v, (m,) * 6)
        for axis, d in ((2, 0), (1, 1), (0, 2)):
            if self.per[d]:
                c = a.narrow(axis, m, self.n[d])
                a = torch.cat([c.narrow(axis, self.n[d] - m, m), c, c.narrow(axis, 0, m)], axis)
        self.f[name] = a

    def _e(self, h):
        f, i = self.f, self._in
        ix, iy, iz = (1.0 / v for v in self.d)
        bx, by, bz = (i(f[k]) for k in ("bx", "by", "bz"))
        jx, jy, jz = (i(self.r[k], ring=1) for k in ("jx", "jy", "jz"))
        ex = h * ((bz - i(f["bz"], dy=-1)) * iy - (by - i(f["by"], dz=-1)) * iz - jx)
        ey = h * ((bx - i(f["bx"], dz=-1)) * iz - (bz - i(f["bz"], dx=-1)) * ix - jy)
        ez = h * ((by - i(f["by"], dx=-1)) * ix - (bx - i(f["bx"], dy=-1)) * iy - jz)
        for k, v in (("ex", ex), ("ey", ey), ("ez", ez)):
            self._add(k, v)

    def _b(self, h):
        f, i = self.f, self._in
        ix, iy, iz = (1.0 / v for v in self.d)
        ex, ey, ez = (i(f[k]) for k in ("ex", "ey", "ez"))
        bx = -h * ((i(f["ez"], dy=1) - ez) * iy - (i(f["ey"], dz=1) - ey) * iz)
        by = -h * ((i(f["ex"], dz=1) - ex) * iz - (i(f["ez"], dx=1) - ez) * ix)
        bz = -h * ((i(f["ey"], dx=1) - ey) * ix - (i(f["ex"], dy=1) - ex) * iy)
        for k, v in (("bx", bx), ("by", by), ("bz", bz)):
            self._add(k, v)

    def _set(self, name, axis, at, v):
        """one plane of a field (physical rows of the other axes) set to v"""
        a = self.f[name].clone()
        m, sl = self.m, [None] * 3
        for ax, d in ((2, 0), (1, 1), (0, 2)):
            sl[ax] = at if ax == axis else slice(m, m + self.n[d])
        a[tuple(sl)] = v
        self.f[name] = a

    def _source(self, time):
        """-envelope x transverse amplitude x cos(phase) at x = 0, (nz, ny)"""
        m, (nx, ny, nz) = self.m, self.n
        L = [n * h for n, h in zip(self.n, self.d)]
        k = 2 * PI / LAMBDA
        rl = 0.5 * k * self.waist ** 2
        xe = -0.5 * L[0]
        y = (torch.arange(ny, dtype=torch.float64, device=self.dev) + m) * self.d[1] - 0.5 * L[1]
        z = (torch.arange(nz, dtype=torch.float64, device=self.dev) + m) * self.d[2] - 0.5 * L[2]
        r2 = y[None, :] ** 2 + z[:, None] ** 2
        w = self.waist * math.sqrt(1 + (xe / rl) ** 2)
        phi = (xe / rl) * r2 / w / w - math.atan(xe / rl) + k * xe - time
        t = time - self.start
        dur = 10.0 * LAMBDA
        if self.absorbing:
            env = self.amp * math.exp(-2 * math.log(2) * ((t - 1.5 * dur) / dur) ** 2) if 0 <= t <= 3 * dur else 0.0
        else:
            env = self.amp * math.sin(PI * t / dur) if 0 <= t <= dur else 0.0
        if self.coef is not None:
            nc = self.coef.shape[0]

            def basis(n):
                u = (torch.arange(n, dtype=torch.float64, device=self.dev) + 0.5) / n * (nc - 1)
                a = (u[:, None] - torch.arange(nc, dtype=torch.float64, device=self.dev)[None, :]).abs()
                return torch.where(a < 1, (4 - 6 * a ** 2 + 3 * a ** 3) / 6, (2 - a).clamp(min=0) ** 3 / 6)

            amp = basis(nz) @ self.coef @ basis(ny).T
        else:
            amp = self.waist / w * torch.exp(-r2 / (w * w))
        return -env * amp * torch.cos(phi + self.phase)

    def _boundary(self, step):
        m, dt = self.m, self.dt
        if not self.per[0]:
            hx, hy, hz = (dt / h for h in self.d)
            al, be = 1 / (1 + hx), 1 - hx
            src = self._source(step * dt) if self.amp else 0.0
            for side, col, out in ((0, m, m - 1), (1, self.n[0], self.n[0] + 1)):
                if side == 1 and self.absorbing:
                    continue
                f = {k: self._in(self.f[k], dx=col - m)[:, :, 0] for k in FIELDS}
                bx = f["bx"]
                bxz, bxy = (self._in(self.f["bx"], dx=col - m, **q)[:, :, 0] for q in (dict(dz=-1), dict(dy=-1)))
                jy, jz = (self._in(self.r[k], dx=col - m, ring=1)[:, :, 0] for k in ("jy", "jz"))
                sg = 1.0 if side == 0 else -1.0
                s = 4 * src if side == 0 else 0.0
                bz = al * (s - sg * 2 * f["ey"] - hz * (bx - bxz) - be * f["bz"] - sg * dt * jy)
                by = al * (sg * 2 * f["ez"] + hy * (bx - bxy) - be * f["by"] + sg * dt * jz)
                self._set("bz", 2, out, bz)
                self._set("by", 2, out, by)
        if not self.absorbing:
            return
        for axis, d, lo in ((1, 1, 1), (1, 1, 0), (0, 2, 1), (0, 2, 0), (2, 0, 0)):
            h = dt / self.d[d]
            al, be, sg = 1 / (1 + h), 1 - h, 1.0 if lo else -1.0
            row = m if lo else self.n[d] + m - 1
            tgt, inn = (row - 1, row) if lo else (row, row - 1)

            def at(name, q, ring=0):
                a = self.r[name] if ring else self.f[name]
                sl = [None] * 3
                for ax, dd in ((2, 0), (1, 1), (0, 2)):
                    sl[ax] = q + ring if ax == axis else slice(m + ring, m + ring + self.n[dd])
                return a[tuple(sl)]

            one, two = {1: (("bx", "ez", "jz"), ("bz", "ex", "jx")), 0: (("by", "ex", "jx"), ("bx", "ey", "jy")),
                        2: (("bz", "ey", "jy"), ("by", "ez", "jz"))}[axis]
            v1 = al * (sg * (-2 * at(one[1], row) - dt * at(one[2], row, 1)) - be * at(one[0], inn))
            v2 = al * (sg * (2 * at(two[1], row) + dt * at(two[2], row, 1)) - be * at(two[0], inn))
            self._set(one[0], axis, tgt, v1)
            self._set(two[0], axis, tgt, v2)

    def _fold(self):
        """every ring point becomes the sum over its periodic images"""
        m = self.m
        for name in RINGS:
            a = self.r[name]
            for axis, d in ((2, 0), (1, 1), (0, 2)):
                if not self.per[d]:
                    continue
                n, size = self.n[d], a.shape[axis]
                low, high = m + 1, m + 1   # ghosts below and above the physical points
                c = a.narrow(axis, low, n)
                add = torch.zeros_like(c)
                add.narrow(axis, n - low, low).add_(a.narrow(axis, 0, low))
                add.narrow(axis, 0, high).add_(a.narrow(axis, low + n, high))
                c = c + add
                a = torch.cat([c.narrow(axis, n - low, low), c, c.narrow(axis, 0, size - n - low)], axis)
            self.r[name] = a

    # -- particles ---------------------------------------------------------
    def _gather(self, name, base, wx, wy, wz):
        a = self.f[name]
        sy, sz = a.shape[2], a.shape[1] * a.shape[2]
        flat, P = a.reshape(-1), self.order + 1
        i0 = (base[:, 2] * sz + base[:, 1] * sy + base[:, 0])[:, None] + torch.arange(P, device=self.dev)[None, :]
        tot = 0
        for k in range(P):
            for j in range(P):
                tot = tot + wz[:, k] * wy[:, j] * (wx * flat[i0 + (k * sz + j * sy)]).sum(1)
        return tot

    def _push_some(self, kind, x, p, w, cur):
        """new positions and momenta of some particles of a species, their
        current and charge added into the flat arrays `cur`"""
        P, H, m, n = self.order + 1, self.order // 2, self.m, self.n
        dt, h = self.dt, self.d
        wrapped = []
        for d in range(3):
            v = x[:, d]
            if self.per[d]:
                v = torch.where(v < 0, v + n[d], v)
                v = torch.where(v > n[d], v - n[d], v)
            wrapped.append(v)
        x = torch.stack(wrapped, 1)
        xc = x + (m - 1)
        ip, idd = (xc.detach() + 0.5).floor().long(), xc.detach().floor().long()
        dp, dd = xc - ip, xc - 0.5 - idd
        wp = [_weights(dp[:, d], self.order) for d in range(3)]
        wd = [_weights(dd[:, d], self.order) for d in range(3)]
        e, b = [], []
        for c, dual in (("ex", (1, 0, 0)), ("ey", (0, 1, 0)), ("ez", (0, 0, 1)), ("bx", (0, 1, 1)), ("by", (1, 0, 1)),
                        ("bz", (1, 1, 0))):
            base = torch.stack([(idd if dual[d] else ip)[:, d] - H for d in range(3)], 1)
            v = self._gather(c, base, *[(wd if dual[d] else wp)[d] for d in range(3)])
            (e if c[0] == "e" else b).append(v)
        qm = CHARGE[kind] / MASS[kind] * dt / 2
        e, b = torch.stack(e, 1) * qm, torch.stack(b, 1) * qm
        p1 = p + e
        t = b / torch.sqrt(1 + (p1 * p1).sum(1, keepdim=True))
        s = 2 * t / (1 + (t * t).sum(1, keepdim=True))
        p2 = p1 + torch.linalg.cross(p1, t)
        pn = p1 + torch.linalg.cross(p2, s) + e
        g = torch.sqrt(1 + (pn * pn).sum(1, keepdim=True))
        xn = x + pn / g * dt / torch.tensor(h, dtype=torch.float64, device=self.dev)
        xc2 = xn + (m - 1)
        i2 = (xc2.detach() + 0.5).floor().long()
        d2 = xc2 - i2
        base, s0, ds = [], [], []
        for d in range(3):
            lo = torch.minimum(ip[:, d], i2[:, d])
            base.append(lo - H)
            w0, w1 = wp[d], _weights(d2[:, d], self.order)
            z = torch.zeros_like(w0[:, :1])
            o0, o1 = (ip[:, d] != lo)[:, None], (i2[:, d] != lo)[:, None]
            a0 = torch.where(o0, torch.cat([z, w0], 1), torch.cat([w0, z], 1))
            a1 = torch.where(o1, torch.cat([z, w1], 1), torch.cat([w1, z], 1))
            s0.append(a0)
            ds.append(a1 - a0)
        rs = self.r["jx"].shape
        st = (1, rs[2], rs[1] * rs[2])
        size = rs[0] * rs[1] * rs[2]
        qw = CHARGE[kind] * w
        org = (base[0] + 1) + (base[1] + 1) * st[1] + (base[2] + 1) * st[2]
        for c, (u, v) in enumerate(((1, 2), (0, 2), (0, 1))):
            # the last running sum is the sum of all differences: zero
            a = torch.cumsum(ds[c], 1)[:, :P]
            last = (ip[:, c] == i2[:, c])[:, None] & (torch.arange(P, device=self.dev)[None, :] == P - 1)
            a = torch.where(last, torch.zeros_like(a), a) * (-qw * h[c] / dt)[:, None]
            ia = org[:, None] + torch.arange(P, device=self.dev)[None, :] * st[c]
            for q in range(P + 1):
                for r in range(P + 1):
                    W = (s0[u][:, q] * s0[v][:, r] + 0.5 * ds[u][:, q] * s0[v][:, r] + 0.5 * s0[u][:, q] * ds[v][:, r] +
                         ds[u][:, q] * ds[v][:, r] / 3)
                    cur[c] = cur[c].index_add(0, (ia + (q * st[u] + r * st[v])).clamp(max=size - 1).reshape(-1),
                                              (a * W[:, None]).reshape(-1))
        if self.coef is None:
            org = (i2[:, 0] - H + 1) + (i2[:, 1] - H + 1) * st[1] + (i2[:, 2] - H + 1) * st[2]
            w1 = [_weights(d2[:, d].detach(), self.order) for d in range(3)]
            ia = org[:, None] + torch.arange(P, device=self.dev)[None, :]
            for k in range(P):
                for j in range(P):
                    cur[3 + kind] = cur[3 + kind].index_add(
                        0, (ia + k * st[2] + j * st[1]).reshape(-1),
                        (qw[:, None] * (w1[2][:, k] * w1[1][:, j])[:, None] * w1[0]).reshape(-1))
        return xn, pn

    def push(self):
        cur = [self.r[k].reshape(-1) for k in RINGS]
        for kind in range(2):
            if self.sp[kind] is None or not len(self.sp[kind][2]):
                continue
            x, p, w = self.sp[kind]
            done = [self._push_some(kind, x[o:o + self.CHUNK], p[o:o + self.CHUNK], w[o:o + self.CHUNK], cur)
                    for o in range(0, len(w), self.CHUNK)]
            x, p = torch.cat([v[0] for v in done]), torch.cat([v[1] for v in done])
            keep = torch.ones(len(w), dtype=torch.bool, device=self.dev)
            for d in range(3):
                if not self.per[d]:
                    keep &= (x[:, d].detach() >= 0) & (x[:, d].detach() < self.n[d])
            self.sp[kind] = (x, p, w) if bool(keep.all()) else (x[keep], p[keep], w[keep])
            if self.coef is not None:
                self.alive = self.alive[keep]
        for k, v in zip(RINGS, cur):
            self.r[k] = v.reshape(self.r[k].shape)

    def one_step(self, step):
        self._boundary(step)
        self._e(self.dt / 2)
        self._b(self.dt / 2)
        self.r = {k: torch.zeros_like(v) for k, v in self.r.items()}
        self.push()
        self._fold()
        self._b(self.dt / 2)
        self._e(self.dt / 2)

    def diagnostics(self):
        dv = self.d[0] * self.d[1] * self.d[2]
        en = 0.5 * dv * sum(float((self._in(self.f[k]) ** 2).sum()) for k in FIELDS)
        kin, ch = [0.0, 0.0], [0.0, 0.0]
        for k in range(2):
            x, p, w = self.sp[k]
            u2 = (p * p).sum(1)
            kin[k] = float((w * MASS[k] * u2 / (torch.sqrt(1 + u2) + 1)).sum())
            ch[k] = float(self._in(self.r[RINGS[3 + k]], ring=1).sum()) * dv
        return [en] + kin + ch


def _exact_adjoint(case, seed):
    """loss and gradients by automatic differentiation of the loop, one step
    recomputed at a time"""
    from torch.utils.checkpoint import checkpoint
    knots, coef = _adjoint_inputs(seed)
    n = case["nx"] * case["ny"] * case["nz"] * case["ppc0"]
    c = np.repeat(np.arange(n // case["ppc0"]), case["ppc0"])
    x = np.random.default_rng(seed).random((n, 3)) + np.stack(
        [c % case["nx"], (c // case["nx"]) % case["ny"], c // (case["nx"] * case["ny"])], 1)
    t = np.clip(x[:, 0] / case["nx"] * 31, 0.0, 31 - 1e-12)
    i = np.floor(t).astype(np.int64)
    w0 = ((1 - (t - i)) * knots[i] + (t - i) * knots[i + 1]) / case["ppc0"]
    cf = torch.as_tensor(coef).requires_grad_()
    loop = _Loop(case, seed, coef=cf)
    cf_dev = cf.to(loop.dev)
    w = loop.t(w0).requires_grad_()
    loop.alive = torch.arange(n, device=loop.dev)
    names = FIELDS + RINGS[:3]

    def step(s, alive, coef_, *state):
        loop.coef, loop.alive = coef_, alive
        loop.f = dict(zip(FIELDS, state[:6]))
        loop.r = dict(zip(RINGS, list(state[6:9]) + [loop.r["rho0"], loop.r["rho1"]]))
        loop.sp = [tuple(state[9:12]), None]
        if s == 0:
            loop.push()
        else:
            loop.one_step(s)
        return tuple(loop.f[k] for k in FIELDS) + tuple(loop.r[k] for k in RINGS[:3]) + loop.sp[0] + (loop.alive,)

    state = tuple(loop.f[k] for k in FIELDS) + tuple(loop.r[k] for k in RINGS[:3]) + (
        loop.t(x), torch.zeros((n, 3), dtype=torch.float64, device=loop.dev), w)
    alive = loop.alive
    for s in range(case["steps"] + 1):
        out = checkpoint(step, s, alive, cf_dev, *state, use_reentrant=False)
        state, alive = out[:-1], out[-1]
    xs, ps, ws = state[len(names):]
    lo, hi = _window(case)
    up, down = (xs[:, 0] - lo) / 2.0, (hi - xs[:, 0]) / 2.0
    win = torch.where(up < 1, torch.sin(0.5 * math.pi * up) ** 2, torch.ones_like(up)) * torch.where(
        down < 1, torch.sin(0.5 * math.pi * down) ** 2, torch.ones_like(up))
    win = torch.where((xs[:, 0] >= lo) & (xs[:, 0] < hi), win, torch.zeros_like(win))
    u2 = (ps * ps).sum(1)
    loss = (win * ws * u2 / (torch.sqrt(1 + u2) + 1)).sum()
    loss.backward()
    return {"loss": float(loss.detach()), "weights": w.grad.cpu(), "profile": cf.grad.reshape(-1)}
