"""Rounding of the FP32 push and deposit.

FP32 contexts round at every operation; what they may not do is to round more
than the plain form of the same arithmetic in single precision.

* Momenta: the Boris step written with IEEE square root and divisions and fused
  half kicks (numpy, float32) against the same step in double gives the error
  to stay within, on the same particles; both are root-mean-square over 60,000
  particles, so that chance differences are below 1 %, and 3 % is allowed.
* Sums: N equal particles of a node deposit N/2 times the current of two.  The
  accumulators are exact; what is left is the rounding of the two results to
  24 bits (2^-24 each) and of one particle's share to the accumulators' step
  (at the points compared, over 2^24 steps high, below 2^-25), so that the two
  agree to 2^-23 + 2^-25 at every point.  The weight makes the accumulators'
  scale a power of two, whose product rounds nothing.  (Two, not one: a particle
  that is alone in its row is deposited in another way at 4th order.)
* rho at 2nd order: the new shapes evaluated at the new offset and their
  products in float32 (numpy) give the error to stay within, root mean square
  over some 4,000 points; 3 % is allowed.  A heavier particle elsewhere makes
  the scale a power of two.
"""
import numpy as np
import pytest

import oracle as O
from pic3d_b200 import workloads as W

pytestmark = pytest.mark.gpu

F = np.float32


def boris(p, e, b, qm, rt):
    """the Boris step in precision rt; the half kicks are fused multiply-adds
    (the product and the sum in double, rounded once)"""
    p, b, qm = p.astype(rt), b.astype(rt), rt(qm)

    def cross(a, c):
        return np.stack([a[1] * c[2] - a[2] * c[1], a[2] * c[0] - a[0] * c[2], a[0] * c[1] - a[1] * c[0]])

    def kick(a):
        return (a.astype(np.float64) + (e * np.float64(qm))[:, None]).astype(rt)
    p1 = kick(p)
    t = (b * qm)[:, None] / np.sqrt(rt(1) + (p1[0] * p1[0] + p1[1] * p1[1] + p1[2] * p1[2]))
    s = t * (rt(2) / (rt(1) + t[0] * t[0] + t[1] * t[1] + t[2] * t[2]))
    p2 = p1 + cross(p1, t)
    return kick(p1 + cross(p2, s))


@pytest.mark.parametrize("size", [1e-3, 0.1, 1.0, 30.0])
def test_momenta_round_no_more_than_square_root_and_division(size):
    from pic3d_b200.simulation import Simulation
    w = W.Workload(name="boris", nx=12, ny=12, nz=12, mem=2, period=(1, 1, 1), ppc=(1, 0), steps=1)
    n, qm = 20000, -w.params()["dt_half"]
    err = {"gpu": 0.0, "plain": 0.0}
    for seed in range(3):
        rng = np.random.default_rng(seed)
        eb = np.round(64 * rng.uniform(-1.0, 1.0, 6)) / 64
        p = (size * rng.normal(size=(3, n))).astype(F).astype(np.float64)
        rec = np.zeros(n, dtype=W.PARTICLE_DTYPE)
        rec["id"] = np.arange(n)
        for d, f in enumerate("xyz"):
            rec[f] = rng.integers(0, 12, n)   # whole cells: shapes and gather are exact
            rec["p" + f] = p[d]
        rec["charge"], rec["mass"], rec["weight"] = -1.0, 1.0, 0.1
        sim = Simulation(w, precision="fp32")
        sim.upload_particles(0, rec)
        for c, name in enumerate(("ex", "ey", "ez", "bx", "by", "bz")):
            sim.upload_array(name, np.full(sim.field_shape(), eb[c]))
        sim.clear_currents()
        sim.update_particle_position_momentum(0)
        out = np.sort(sim.download_particles(0), order="id")
        sim.close()
        ref = boris(p, eb[:3], eb[3:], float(F(qm)), np.float64)
        norm = np.sum(ref ** 2, axis=0)
        got = np.stack([out["px"], out["py"], out["pz"]])
        err["gpu"] += np.mean(np.sum((got - ref) ** 2, axis=0) / norm)
        err["plain"] += np.mean(np.sum((boris(p, eb[:3], eb[3:], F(qm), F) - ref) ** 2, axis=0) / norm)
    assert err["gpu"] <= 1.03 ** 2 * err["plain"], {k: np.sqrt(v / 3) for k, v in err.items()}


@pytest.mark.parametrize("mem", [2, 4], ids=["o2", "o4"])
@pytest.mark.parametrize("count", [7, 32, 75])
def test_equal_particles_add_up_exactly(count, mem):
    from pic3d_b200.simulation import Simulation
    w = W.Workload(name="equal", nx=16, ny=12, nz=10, mem=mem, period=(1, 1, 1), ppc=(1, 0), steps=1)
    weight = w.dt / 1.01   # scale: 2^31 / (1.01 |q w| d / dt)
    worst = 0.0
    for seed in range(8):
        rng = np.random.default_rng(seed)
        p = rng.uniform(-2.0, 2.0, 3)
        move = p / np.sqrt(1 + p @ p) * w.dt
        # node 6 of a tile of nodes 4 .. 7, moving without leaving its node
        x = 6.0 - 0.5 * move + 0.1 * rng.uniform(-1.0, 1.0, 3) * (0.5 - 0.5 * np.abs(move))
        j = []
        for m in (2, count):
            rec = np.zeros(m, dtype=W.PARTICLE_DTYPE)
            rec["id"] = np.arange(m)
            for d, f in enumerate("xyz"):
                rec[f], rec["p" + f] = x[d], p[d]
            rec["charge"], rec["mass"], rec["weight"] = -1.0, 1.0, weight
            sim = Simulation(w, precision="fp32")
            sim.upload_particles(0, rec)
            sim.clear_currents()
            sim.update_particle_position_momentum(0)
            j.append(np.stack([sim.download_array(a) for a in ("jx", "jy", "jz")]))
            sim.close()
        big = np.abs(j[0]) / 2 >= 2.0 ** -7   # 2^24 steps
        assert big.sum() > 4
        worst = max(worst, float(np.max(np.abs(2.0 * j[1][big] / j[0][big] / count - 1.0))))
    assert worst <= 2.0 ** -23 + 2.0 ** -25, worst


def test_rho_rounds_no_more_than_its_shapes_do():
    from pic3d_b200.simulation import Simulation
    n = (32, 24, 24)
    w = W.Workload(name="rho", nx=n[0], ny=n[1], nz=n[2], mem=2, period=(1, 1, 1), ppc=(1, 0), steps=1)
    rng = np.random.default_rng(12)
    m = 8000
    rec = np.zeros(m, dtype=W.PARTICLE_DTYPE)
    rec["id"] = np.arange(m)
    cell, off, p = [], [], []
    for d, f in enumerate("xyz"):
        # nodes 1 .. 3 of every other tile, so that no point gets the (rounded) sums of two
        cell.append(8 * rng.integers(0, n[d] // 8, m) + 1 + rng.integers(0, 2, m))
        off.append(np.minimum(rng.random(m), 0.999).astype(F))
        p.append((0.3 * rng.normal(size=m)).astype(F))
        rec[f], rec["p" + f] = cell[d] + off[d].astype(np.float64), p[d]
    rec["gamma"] = np.sqrt(1 + rec["px"] ** 2 + rec["py"] ** 2 + rec["pz"] ** 2)
    rec["charge"], rec["mass"], rec["weight"] = -1.0, 1.0, 1.0
    none = np.zeros(0, dtype=W.PARTICLE_DTYPE)
    heavy = rec[:1].copy()
    heavy["id"], heavy["weight"], heavy["gamma"] = m, 1.0 / (1.01 * 0.75 ** 3), 1.0   # scale: 2^31 / (1.01 |q w| (3/4)^3)
    for f in "xyz":
        heavy[f], heavy["p" + f] = 14.0, 0.0
    both = np.zeros(m + 1, dtype=W.PARTICLE_DTYPE)
    both[:m], both[m:] = rec, heavy
    g = w.mem + 1
    inner = tuple(slice(g, g + n[d]) for d in (2, 1, 0))
    rho = []
    for parts in (rec, heavy):
        o = O.Oracle(w, [parts, none])
        o.step(1)
        rho.append(o.state()["rho0"][inner])
    want, there = rho[0], rho[1] == 0.0

    node, shapes = [], []
    for d in range(3):
        e = (p[d] / rec["gamma"] * w.dt).astype(F)
        d0 = np.where(off[d] >= F(0.5), off[d] - F(1), off[d])
        d1 = d0 + e
        cross = np.where(d1 >= F(0.5), 1, np.where(d1 < F(-0.5), -1, 0))
        t1 = e - (F(0.5) * cross.astype(F) - d0)     # past the knot
        d1 = np.where(cross == 0, d1, t1 - F(0.5) * cross.astype(F))
        node.append(cell[d] + (off[d] >= F(0.5)) + cross)
        h = F(0.5)
        mid = (0.75 - d1.astype(np.float64) ** 2).astype(F)   # a fused multiply-add
        shapes.append((h * (h - d1) * (h - d1), mid, h * (h + d1) * (h + d1)))
    plain = np.zeros(n[::-1])
    for k in range(3):
        wk = -shapes[2][k]
        for j in range(3):
            wjk = wk * shapes[1][j]
            for i in range(3):
                np.add.at(plain, ((node[2] + k - 1) % n[2], (node[1] + j - 1) % n[1], (node[0] + i - 1) % n[0]),
                          (wjk * shapes[0][i]).astype(np.float64))
    # index of node 0 in the array: the point the oracle's rho agrees at
    shift = [s for s in np.ndindex(3, 3, 3)
             if np.allclose(np.roll(plain, [q - 1 for q in s], (0, 1, 2)), want, rtol=0, atol=1e-5 * np.abs(want).max())]
    assert len(shift) == 1
    plain = np.roll(plain, [q - 1 for q in shift[0]], (0, 1, 2))

    sim = Simulation(w, precision="fp32")
    sim.upload_particles(0, both)
    sim.run_main_time_loop(1)
    got = sim.download_array("rho0")[inner]
    sim.close()
    err = {k: np.linalg.norm((a - want)[there]) / np.linalg.norm(want[there]) for k, a in (("gpu", got), ("plain", plain.astype(F)))}
    assert err["gpu"] <= 1.03 * err["plain"], err
