"""Tiles of nodes at the number of particles their accumulators hold.

A tile with up to 16383 particles of both species is pushed by its CTA from
shared memory; one more and the whole tile goes to the global kernel.  The
particles lie in nodes 0 .. 3 of every axis (positions up to 3.4), spread over
the tile, or all in one node and flying the same way, where the limbs of the
accumulators come closest to their limits.  One step against the oracle at the
one-step parity bounds, and the count that the global kernel took.
"""
import numpy as np
import pytest

import oracle as O
from parity import TOL_FP32, TOL_FP64, array_errors, particle_errors, periods

from pic3d_b200 import workloads as W

pytestmark = pytest.mark.gpu

LIMIT = 16383


def electrons(n, spread, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros(n, dtype=W.PARTICLE_DTYPE)
    p["id"] = np.arange(n)
    for d, f in enumerate("xyz"):
        p[f] = 0.05 + 3.35 * rng.random(n) if spread == "tile" else 2.0 + 0.2 * (rng.random(n) - 0.5)
        p["p" + f] = 0.1 * rng.normal(size=n) if spread == "tile" else (0.2, 0.15, -0.1)[d]
    p["gamma"] = np.sqrt(1 + p["px"] ** 2 + p["py"] ** 2 + p["pz"] ** 2)
    p["charge"], p["mass"], p["weight"] = -1.0, 1.0, 0.01
    return p


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mem", [2, 4], ids=["o2", "o4"])
@pytest.mark.parametrize("spread", ["tile", "one_node"])
@pytest.mark.parametrize("extra", [0, 1], ids=["full", "over_full"])
def test_a_full_tile_matches_the_oracle(extra, spread, mem, precision):
    from pic3d_b200.simulation import Simulation
    w = W.Workload(name="full", nx=16, ny=12, nz=10, mem=mem, period=(1, 1, 1), ppc=(1, 0), u_th=(0.1, 0.0), steps=1)
    parts = [electrons(LIMIT + extra, spread, seed=3), np.zeros(0, dtype=W.PARTICLE_DTYPE)]
    o = O.Oracle(w, parts)
    o.step(1)
    ref = o.state()
    sim = Simulation(w, precision=precision)
    sim.upload_particles(0, parts[0])
    sim.run_main_time_loop(1)
    by_global = sim.particle_order_stats(0)["global_kernel"]
    got = sim.state()
    sim.close()
    assert by_global == (LIMIT + 1 if extra else 0)
    tol, pos_tol = (TOL_FP64, 1e-11) if precision == "fp64" else (TOL_FP32, 2e-6)
    errs = array_errors(got, ref)
    assert max(errs.values()) < tol, errs
    perr, merr = particle_errors(got["particles"][0], ref["particles"][0], periods(w.params()))
    assert perr < pos_tol and merr < tol, (perr, merr)
