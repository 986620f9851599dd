"""Rounding of the FP32 push.

FP32 contexts round at every operation; what they may not do is to round more
than the plain form of the same arithmetic in single precision.

* Momenta: the Boris step written with IEEE square root and divisions and fused
  half kicks (numpy, float32) against the same step in double gives the error
  to stay within, on the same particles; both are root-mean-square over 60,000
  particles, so that chance differences are below 1 %, and 3 % is allowed.
"""
import numpy as np
import pytest

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
